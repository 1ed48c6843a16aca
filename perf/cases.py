"""Timed work of the library: what its users have it compute, through its
public entry points, from the smallest calls to the largest.

Kinds of cases:
  grid    scarf_initialize + scarf_execute of the spectral representation
          method (SRM) on a structured 2-D or 3-D grid, into a device field or
          an ordinary (pageable) host array
  points  the same on an unstructured point set
  fim     scarf_execute of the Fourier integral method on a structured grid
  direct  the FP32 direct sum over device points and a harmonic table
  tc      the tensor-core sum of one structured block from a harmonic table
  batch   many uneven fields in one tensor-core launch

Every pass of an execute case draws its harmonics anew from its seed, as the
library's users have it: a mesh is set up once and one field is drawn per
seed. The direct, tc and batch cases are the building blocks that programs
with their own harmonic tables call.
"""
import ctypes
import math

import numpy as np
import torch

import scarf3d_b200 as sb

VK, GS = 0, 1  # autocorrelation functions: von Karman, Gaussian


def listed():
    return [
        # A small 2-D test map: latency of one call.
        {"name": "grid2d_small", "kind": "grid", "nx": 96, "ny": 64, "nz": 0, "ds": 50.0, "acf": GS, "hurst": 0.0,
         "cl": 0.1, "nharm": 500, "alpha": 0.0, "post": False, "host": False},
        # A rotated 2-D section at the reference's harmonic count.
        {"name": "grid2d_map", "kind": "grid", "nx": 1201, "ny": 800, "nz": 0, "ds": 50.0, "acf": VK, "hurst": 0.25,
         "cl": 0.05, "nharm": 10000, "alpha": 20.0, "post": False, "host": False},
        # The plain benchmark configuration: 128^3 points at 50 m, 5 000 harmonics.
        {"name": "grid3d_128", "kind": "grid", "nx": 128, "ny": 128, "nz": 128, "ds": 50.0, "acf": VK, "hurst": 0.25,
         "cl": 0.315, "nharm": 5000, "alpha": 0.0, "post": False, "host": False},
        # An uneven, rotated block, rescaled to its sigma and tapered around
        # two points of interest (receivers, a hypocentre).
        {"name": "grid3d_ragged_post", "kind": "grid", "nx": 203, "ny": 151, "nz": 97, "ds": 25.0, "acf": GS,
         "hurst": 0.0, "cl": 0.12, "nharm": 10000, "alpha": 30.0, "post": True, "host": False},
        # A medium model into an ordinary host array (the C API's usual caller).
        {"name": "grid3d_host", "kind": "grid", "nx": 320, "ny": 288, "nz": 200, "ds": 40.0, "acf": VK, "hurst": 0.4,
         "cl": 0.1, "nharm": 10000, "alpha": 0.0, "post": False, "host": True},
        # The headline configuration: 512^3 points at 25 m, 20 000 harmonics.
        {"name": "grid3d_512", "kind": "grid", "nx": 512, "ny": 512, "nz": 512, "ds": 25.0, "acf": VK, "hurst": 0.5,
         "cl": 0.2348, "nharm": 20000, "alpha": 0.0, "post": False, "host": False},
        # A receiver network or a coarse mesh: few points, every harmonic.
        {"name": "points_few", "kind": "points", "npts": 5003, "dh": 100.0, "acf": GS, "hurst": 0.0, "nharm": 10000},
        # The unstructured benchmark configuration: 2e6 mesh points, 10 000 harmonics.
        {"name": "points_2m", "kind": "points", "npts": 2000000, "dh": 100.0, "acf": GS, "hurst": 0.0,
         "nharm": 10000},
        # Device points and a table in hand: one mesh partition.
        {"name": "direct_block", "kind": "direct", "npts": 150001, "dh": 100.0, "hurst": 0.25, "nharm": 4000},
        # One structured block from a table in hand.
        {"name": "tc_block", "kind": "tc", "nx": 256, "ny": 192, "nz": 160, "ds": 25.0, "hurst": 0.5, "nharm": 8000},
        # Many realisations at once: uneven grids and harmonic counts.
        {"name": "tc_batch", "kind": "batch", "fields": 48, "axis_max": 256, "nharm_max": 20000, "hurst": 0.4},
        # The Fourier integral method on the headline grid.
        {"name": "fim_512", "kind": "fim", "nx": 512, "ny": 512, "nz": 512, "ds": 25.0, "acf": VK, "hurst": 0.5,
         "cl": 0.1, "pad": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# point x harmonic pairs of the largest listed case (512^3 x 20 000), and of
# the largest direct sum over points (2e6 x 10 000)
_MOST_GRID, _MOST_POINTS = 512**3 * 20000, 2000000 * 10000


def draw(rng):
    kind = rng.choice(["grid2d", "grid3d", "grid3d", "grid3d", "points", "points", "direct", "tc", "batch", "fim"])
    acf = rng.choice([VK, GS])
    hurst = round(rng.uniform(0.1, 0.9), 3) if acf == VK else 0.0
    ds = rng.choice([10.0, 25.0, 40.0, 50.0, 100.0])
    if kind in ("grid2d", "grid3d"):
        while True:
            nx, ny = _log(rng, 48, 1600), _log(rng, 48, 1600)
            nz = 0
            if kind == "grid3d":
                nx, ny, nz = _log(rng, 32, 512), _log(rng, 32, 512), _log(rng, 32, 512)
            nharm = _log(rng, 500 if kind == "grid2d" else 1000, 20000)
            if nx * ny * max(nz, 1) * nharm <= _MOST_GRID:
                break
        host = kind == "grid3d" and nx * ny * nz <= 320 * 288 * 200 and rng.random() < 0.25
        return {"kind": "grid", "nx": nx, "ny": ny, "nz": nz, "ds": ds, "acf": acf, "hurst": hurst,
                "cl": round(rng.uniform(0.06, 0.25), 3), "nharm": nharm,
                "alpha": rng.choice([0.0, 0.0, 15.0, -40.0]), "post": rng.random() < 0.3, "host": host}
    if kind == "points":
        npts = _log(rng, 1000, 2000000)
        nharm = _log(rng, 1000, 10000)
        return {"kind": "points", "npts": npts, "dh": rng.choice([50.0, 100.0, 200.0]), "acf": acf, "hurst": hurst,
                "nharm": nharm}
    hurst = round(rng.uniform(0.1, 0.9), 3)
    if kind == "direct":
        return {"kind": "direct", "npts": _log(rng, 3000, 300000), "dh": rng.choice([50.0, 100.0, 200.0]),
                "hurst": hurst, "nharm": _log(rng, 1000, 8000)}
    if kind == "tc":
        return {"kind": "tc", "nx": _log(rng, 40, 320), "ny": _log(rng, 40, 320), "nz": _log(rng, 40, 320), "ds": ds,
                "hurst": hurst, "nharm": _log(rng, 1000, 12000)}
    if kind == "batch":
        return {"kind": "batch", "fields": rng.randint(8, 48), "axis_max": rng.choice([96, 128, 192, 256]),
                "nharm_max": rng.choice([5000, 10000, 20000]), "hurst": hurst}
    return {"kind": "fim", "nx": _log(rng, 48, 512), "ny": _log(rng, 48, 512), "nz": _log(rng, 48, 400), "ds": ds,
            "acf": acf, "hurst": round(rng.uniform(0.1, 0.9), 3) if acf == VK else 0.0,
            "cl": round(rng.uniform(0.03, 0.2), 3), "pad": rng.random() < 0.3}


# ---------------------------------------------------------------- inputs --
def _extent(c):
    return [c["nx"], c["ny"]] + ([c["nz"]] if c["nz"] else [])


class _Mesh:
    """A mesh in a library context of its own, and its field."""

    def __init__(self, nharm, seed, field, **kw):
        self.ctx, self.seed, self.field = sb.Context(), int(seed), field
        with self.ctx:
            sb.set_nharm(nharm)
            sb.scarf_initialize(**kw)

    def run(self):
        with self.ctx:
            _, stats = sb.scarf_execute(self.seed, self.field)
        # domain flags, standard deviation and mean (the rest are timings)
        return {"field": self.field, "stats": stats[:4]}


def _grid(c, seed):
    n, ds = _extent(c), c["ds"]
    span = [(v - 1) * ds for v in n]
    # a correlation length per axis, with the usual shorter vertical one; the
    # grid's extent over them sets the lowest wavenumber drawn
    cl = [c["cl"] * s for s in span]
    kw = dict(fs=[1] * len(n), fe=n, ds=ds, acf=c["acf"], cl=cl, sigma=0.05, hurst=c["hurst"])
    if c["kind"] == "fim":
        kw.update(method=0, pad=int(c["pad"]))
        nharm = 10000  # unused by this method
    else:
        kw.update(method=1, alpha=c["alpha"])
        nharm = c["nharm"]
        if c["post"]:
            short = min(span)
            poi = np.array([[0.25 * s for s in span], [0.6 * s for s in span]], np.float32)
            kw.update(rescale=1, poi=poi, mute=0.05 * short, taper=0.15 * short)
    npts = int(np.prod(n))
    field = np.zeros(npts, np.float32) if c.get("host") else torch.zeros(npts, device="cuda")
    return _Mesh(nharm, seed, field, **kw)


_BOX = (20000.0, 20000.0, 10000.0)


def _points(c, seed):
    rng = np.random.default_rng(seed)
    x, y, z = ((rng.random(c["npts"], dtype=np.float32) * np.float32(b)) for b in _BOX)
    return _Mesh(c["nharm"], seed, torch.zeros(c["npts"], device="cuda"), x=x, y=y, z=z, dh=c["dh"], acf=c["acf"],
                 cl=[1500.0, 1500.0, 500.0], sigma=0.1, hurst=c["hurst"], method=1)


def _table(rng, nharm, hurst, cl, kmin, kmax):
    """nharm rows {v1, v2, v3, a, b}: wavenumbers of a von Karman spectrum
    between kmin and kmax (in inverse correlation lengths), directions
    uniform on the sphere, normal amplitudes."""
    k = np.exp(np.linspace(math.log(kmin), math.log(kmax), 4097))
    pdf = k**3 * (1.0 + k * k) ** -(hurst + 1.5)  # per unit log k
    cdf = np.concatenate([[0.0], np.cumsum(0.5 * (pdf[1:] + pdf[:-1]))])
    u = np.interp(rng.random(nharm) * cdf[-1], cdf, k)
    phi, cos_t = 2 * math.pi * rng.random(nharm), 1.0 - 2.0 * rng.random(nharm)
    sin_t = np.sqrt(1.0 - cos_t**2)
    v = np.stack([u * np.sin(phi) * sin_t / cl[0], u * np.cos(phi) * sin_t / cl[1], u * cos_t / cl[2]], 1)
    return np.concatenate([v, rng.standard_normal((nharm, 2))], 1).astype(np.float32)


def _setup(nharm, angle_deg, bar):
    """The derived scalars that the summing entry points read."""
    s = sb.SrmSetup()
    t = math.radians(angle_deg)
    m = [math.cos(t), math.sin(t), 0.0, -math.sin(t), math.cos(t), 0.0, 0.0, 0.0, 1.0]
    s.ndim, s.scaling = 3, 0.05 / math.sqrt(nharm)
    for i in range(9):
        s.m[i] = m[i]
    for i in range(3):
        s.bar[i] = bar[i]
    return s


def _i3(v):
    return (ctypes.c_int * 3)(*[int(x) for x in v])


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _direct_inputs(c, seed):
    rng = np.random.default_rng(seed)
    xyz = np.stack([rng.random(c["npts"]) * b for b in _BOX]).astype(np.float32)
    cl = (1500.0, 1500.0, 500.0)
    kmin, kmax = 2 * math.pi * max(a / b for a, b in zip(cl, _BOX)), math.pi / c["dh"] * min(cl)
    return xyz, _table(rng, c["nharm"], c["hurst"], cl, kmin, kmax), _setup(c["nharm"], 20.0, (0.0, 0.0, 0.0))


def _block_inputs(n, ds, hurst, nharm, rng, angle):
    span = [v * ds for v in n]
    cl = [0.2 * s for s in span]
    tab = _table(rng, nharm, hurst, cl, 2 * math.pi * 0.2, math.pi / ds * min(cl))
    return tab, _setup(nharm, angle, (0.5 * span[0], 0.5 * span[1], 0.0))


def _batch_inputs(c, seed):
    """Grid axes log-uniform from 32 points, in multiples of 16 (2 000
    harmonics and up), at 50 m. The shapes belong to the case, not to the
    seed: only the tables change from seed to seed."""
    shape = np.random.default_rng(c["fields"] * 1000 + c["axis_max"])
    rng = np.random.default_rng(seed)
    out = []
    for f in range(c["fields"]):
        n = [int(max(32, round(v / 16) * 16)) for v in np.exp(shape.uniform(math.log(32), math.log(c["axis_max"]), 3))]
        nharm = int(shape.integers(2000, c["nharm_max"] + 1))
        out.append((n, 50.0) + _block_inputs(n, 50.0, c["hurst"], nharm, rng, 10.0 * (f % 3)))
    return out


class _Direct:
    def __init__(self, c, seed):
        xyz, tab, self.s = _direct_inputs(c, seed)
        self.xyz, self.tab = torch.from_numpy(xyz).cuda(), torch.from_numpy(tab).cuda()
        self.field = torch.zeros(c["npts"], device="cuda")

    def run(self):
        x, y, z = self.xyz
        sb.check(sb.lib.scarf_srm_direct_points(ctypes.byref(self.s), _p(x), _p(y), _p(z), x.numel(), _p(self.tab),
                                                len(self.tab), _p(self.field), None))
        return self.field


class _Block:
    def __init__(self, c, seed):
        self.n = [c["nx"], c["ny"], c["nz"]]
        tab, self.s = _block_inputs(self.n, c["ds"], c["hurst"], c["nharm"], np.random.default_rng(seed), 20.0)
        self.ds, self.tab = c["ds"], torch.from_numpy(tab).cuda()
        self.field = torch.zeros(int(np.prod(self.n)), device="cuda")
        self.bytes = sb.tc_workspace_bytes(3, self.n, len(tab))
        self.work = torch.empty(self.bytes, dtype=torch.uint8, device="cuda")

    def run(self):
        sb.check(sb.lib.scarf_srm_tc_structured(ctypes.byref(self.s), _i3([1, 1, 1]), _i3(self.n), self.ds,
                                                _p(self.tab), len(self.tab), _p(self.field), _p(self.work),
                                                self.bytes, None))
        return self.field


class _Batch:
    def __init__(self, c, seed):
        self.tabs, self.fields, entries = [], [], []
        for n, ds, tab, s in _batch_inputs(c, seed):
            self.tabs.append(torch.from_numpy(tab).cuda())
            self.fields.append(torch.zeros(int(np.prod(n)), device="cuda"))
            entries.append(dict(setup=s, fs=[1, 1, 1], n=n, ds=ds, d_table=self.tabs[-1].data_ptr(), nh=len(tab),
                                d_field=self.fields[-1].data_ptr()))
        self.batch = sb.TcBatch(entries, lambda b: torch.empty(b, dtype=torch.uint8, device="cuda"))

    def run(self):
        self.batch.launch()
        self.batch.wait()
        return self.fields


_STATES = {"grid": _grid, "fim": _grid, "points": _points, "direct": _Direct, "tc": _Block, "batch": _Batch}


def prepare(case, seed):
    return _STATES[case["kind"]](case, seed)


def run(state):
    return state.run()


# ------------------------------------------------------------------ work --
def work(case):
    """Each output value is written once and each table or coordinate read
    once. A sum over a regular grid is a Fourier sum, for which 2.5 n log2 n
    operations for the n real values (a fast transform) and a few hundred per
    harmonic do; over scattered points every point and harmonic meet: three
    products and two sums of the phase, its sine and cosine, and their
    weighted sum."""
    def grid(npts, nharm):
        return {"bytes": 4.0 * npts + 20.0 * nharm, "flops": 2.5 * npts * math.log2(max(npts, 2)) + 300.0 * nharm}

    k = case["kind"]
    if k in ("points", "direct"):
        return {"bytes": 16.0 * case["npts"] + 20.0 * case["nharm"], "flops": 11.0 * case["npts"] * case["nharm"]}
    if k == "batch":
        each = [grid(float(np.prod(n)), len(t)) for n, _, t, _ in _batch_inputs(case, 0)]
        return {"bytes": sum(w["bytes"] for w in each), "flops": sum(w["flops"] for w in each)}
    return grid(float(np.prod(_extent(case))), 0 if k == "fim" else case["nharm"])


# ----------------------------------------------------------------- exact --
def _waves(tab, s):
    t = torch.from_numpy(tab).cuda().double()
    m = torch.tensor(list(s.m), dtype=torch.float64, device="cuda").reshape(3, 3)
    bar = torch.tensor(list(s.bar), dtype=torch.float64, device="cuda")
    return t[:, :3] @ m, t[:, :3] @ bar, t[:, 3], t[:, 4]


def _exact_block(n, ds, tab, s):
    k, c, a, b = _waves(tab, s)
    phase = [k[:, d:d + 1] * (torch.arange(n[d], dtype=torch.float64, device="cuda") * ds) for d in range(3)]
    ex = torch.polar(torch.ones_like(phase[0]), phase[0] + c[:, None]) * torch.complex(b, -a)[:, None]
    ey, ez = (torch.polar(torch.ones_like(p), p) for p in phase[1:])
    out = torch.empty(n[2], n[1], n[0], dtype=torch.float64, device="cuda")
    rows = max(1, (1 << 26) // (n[0] * len(tab)))
    for j in range(0, n[1], rows):
        e = (ey[:, j:j + rows, None] * ex[:, None, :]).reshape(len(tab), -1)
        out[:, j:j + rows] = (ez.real.T @ e.real - ez.imag.T @ e.imag).reshape(n[2], -1, n[0])
    return (out * s.scaling).reshape(-1)


def exact(case, seed):
    """The sums from given tables. An executed field has no such value: which
    harmonics it consists of is decided by single-precision comparisons of
    the generator's draws."""
    k = case["kind"]
    if k == "direct":
        xyz, tab, s = _direct_inputs(case, seed)
        kv, c, a, b = _waves(tab, s)
        p = torch.from_numpy(xyz).cuda().double().T
        return torch.cat([torch.sin(t) @ a + torch.cos(t) @ b
                          for t in (q @ kv.T + c for q in p.split(8192))]) * s.scaling
    if k == "tc":
        n = [case["nx"], case["ny"], case["nz"]]
        return _exact_block(n, case["ds"], *_block_inputs(n, case["ds"], case["hurst"], case["nharm"],
                                                          np.random.default_rng(seed), 20.0))
    if k == "batch":
        return [_exact_block(*f) for f in _batch_inputs(case, seed)]
    return None
