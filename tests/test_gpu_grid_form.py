"""The gridded Fourier form that scarf_execute takes for structured meshes
(of enough harmonics for it to be the faster), against the FP64 sum over the same harmonics at every point: grids at the
edges of its plans (one-point and tiny axes, odd sizes, transform lengths of
every radix, several passes over z, tiles past the last plane), rotation, offsets.

Tolerance: the window's interpolation error (nine cells at an oversampling of
1.5: 1.8e-7 rms per transformed axis, up to 1.1e-6 at single wavenumbers) and
FP32 transforms of at most ~12 butterfly levels per axis (~1e-7 sqrt(levels)),
magnified by the window's correction at the grid's edges: below 1e-6 in sum;
2e-6 leaves room for fields of few points, whose rms is one of few values."""
import numpy as np
import pytest

import oracle
import scarf3d_b200 as sb
from oracle import gpu_fp64

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 2e-6


@pytest.fixture(autouse=True)
def _reset():
    yield
    sb.scarf_finalize()
    sb.set_nharm(10000)
    sb.set_form(sb.FORM_AUTO)


def _case(n, nharm, fs=None, acf=0, frac=0.1, angles=(0.0, 0.0, 0.0), ds=25.0, seed=77, dh=None, cl=None):
    fs = fs or [1] * len(n)
    fe = [s + v - 1 for s, v in zip(fs, n)]
    span = max(v - 1 for v in n) * ds
    cl = cl or [max(frac * span, 3 * ds)] * len(n)
    # the domain of the sampler: the largest span along every axis, so that
    # one-point axes do not make the sampling infeasible
    nc, fc = [0.0] * len(n), [span] * len(n)
    kw = dict(acf=acf, hurst=0.4 if acf == 0 else 0.0, sigma=0.05, ds=ds, cl=cl, alpha=angles[0], beta=angles[1],
              gamma=angles[2], dh=dh)
    sb.set_nharm(nharm)
    sb.scarf_initialize(fs=fs, fe=fe, method=1, nc=nc, fc=fc, **kw)
    dev = torch.full((int(np.prod(n)),), float("nan"), device="cuda")
    _, stats = sb.scarf_execute(seed, dev)
    pad = [0.0] * (3 - len(n))
    op = oracle.params(nharm=nharm, seed=seed, nc=nc + pad, fc=fc + pad, **kw)
    so = oracle.setup(op)
    tab, _ = oracle.sample(op, so)
    fs3, n3 = fs + [1] * (3 - len(n)), list(n) + [1] * (3 - len(n))
    ref = gpu_fp64.structured_field(so, fs3, n3, ds, tab)
    rms = float(ref.square().mean().sqrt())
    err = float((dev.double() - ref).square().mean().sqrt()) / rms
    assert err <= TOL, err
    if len(ref) > 1:
        std, mean = float(ref.std()), float(ref.mean())
        assert abs(float(stats[2]) - std) <= 1e-5 * rms and abs(float(stats[3]) - mean) <= 1e-5 * rms
    return dev, stats


@pytest.mark.parametrize("n", [
    (16, 16, 16), (17, 13, 31), (48, 40, 33), (64, 1, 64), (64, 64, 1), (1, 40, 50), (2, 3, 200), (100, 2, 5),
    (31, 97, 65), (200, 9, 3), (128, 81, 32), (333, 20, 40), (20, 251, 40)])
def test_grids_match_fp64(n):
    _case(n, 1500)


@pytest.mark.parametrize("n", [(100, 70), (1201, 40), (37, 801), (5, 300), (300, 1)])
def test_2d_grids_match_fp64(n):
    _case(n, 1500, angles=(20.0, 0.0, 0.0))


@pytest.mark.parametrize("nharm", [1501, 5000, 30000])
def test_harmonic_counts(nharm):
    _case((40, 36, 50), nharm, fs=[5, 3, -7], angles=(30.0, -10.0, 5.0))


@pytest.mark.parametrize("acf,frac,dh", [(1, 0.25, None), (0, 0.25, None), (0, 0.05, 10.0)])
def test_spectra_and_dense_bins(acf, frac, dh):
    # long correlation lengths put most harmonics into a few cells (partial
    # sums); dh < ds keeps wavenumbers up to the grid's Nyquist limit
    _case((96, 80, 64), 6000, acf=acf, frac=frac, dh=dh)


def test_several_passes_and_reproducibility():
    n = (512, 500, 70)  # three passes of 32 planes, the last one partial
    a, sa = _case(n, 3000)
    b, sb_ = _case(n, 3000)
    assert torch.equal(a, b) and np.array_equal(sa[:4], sb_[:4])
    host, sh = sb.scarf_execute(77, np.full(int(np.prod(n)), np.nan, np.float32))
    pinned = torch.full((int(np.prod(n)),), float("nan"), pin_memory=True)
    sb.scarf_execute(77, pinned.numpy())
    assert np.array_equal(host, a.cpu().numpy()) and np.array_equal(pinned.numpy(), host)
    assert np.array_equal(sh[:4], sa[:4])


@pytest.mark.parametrize("n,cl,angles", [
    # correlation lengths that leave the harmonics few of the cells: along x,
    # along y, both, neither; turned; two dimensions
    ((96, 64, 40), (4000.0, 250.0, 250.0), (0.0, 0.0, 0.0)),
    ((96, 64, 40), (250.0, 4000.0, 250.0), (0.0, 0.0, 0.0)),
    ((120, 90, 33), (900.0, 700.0, 200.0), (0.0, 0.0, 0.0)),
    ((48, 40, 36), (300.0, 300.0, 1500.0), (0.0, 0.0, 0.0)),
    ((120, 90, 33), (900.0, 700.0, 200.0), (35.0, -20.0, 50.0)),
    ((30, 200, 33), (300.0, 3000.0, 150.0), (-75.0, 0.0, 0.0)),
    ((300, 140), (2500.0, 300.0), (0.0, 0.0, 0.0)),
    ((140, 300), (300.0, 2500.0), (40.0, 0.0, 0.0)),
])
def test_reach_of_the_harmonics(n, cl, angles):
    _case(n, 3000, cl=list(cl), angles=angles)
