"""The gridded sum with many harmonics in few bins, where blocks rank a bin's
entries: around the line above which they do, bins around the size from which a
block takes one, and entry numbers beyond one bitmap (262 144), against the FP64
sum over the same harmonics, and repeated bit for bit (a wrong or doubled place
loses an entry; an order that depends on arrival changes bits).

Tolerance: the gridded sum's 2e-6 of the field's rms (tests/test_gpu_grid_form.py);
the parts of a bin's sum are FP32, each of at most 32 entries, added in order:
with 300 000 harmonics in a few bins about 1 200 parts, a rounding of at most
sqrt(1200) * 2^-24 = 2e-6 more."""
import numpy as np
import pytest

import oracle
import scarf3d_b200 as sb
from oracle import gpu_fp64

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(40, 36, 33), (90, 70)])
@pytest.mark.parametrize("nharm,frac,tol", [
    (16384, 0.6, 2e-6), (16385, 0.6, 2e-6), (16385, 0.02, 2e-6), (40000, 0.2, 2e-6), (140001, 0.6, 4e-6),
    (300000, 0.5, 4e-6)])
def test_dense_bins_match_fp64(n, nharm, frac, tol):
    ds, seed = 25.0, 11
    span = [(v - 1) * ds for v in n]
    kw = dict(acf=1, hurst=0.0, sigma=0.05, ds=ds, cl=[frac * max(span)] * len(n), alpha=20.0)
    nc, fc = [0.0] * len(n), [max(span)] * len(n)
    sb.set_nharm(nharm)
    try:
        sb.scarf_initialize(fs=[1] * len(n), fe=list(n), method=1, nc=nc, fc=fc, **kw)
        fields = [sb.scarf_execute(seed, torch.full((int(np.prod(n)),), float("nan"), device="cuda"))[0]
                  for _ in range(3)]
    finally:
        sb.scarf_finalize()
        sb.set_nharm(10000)
    assert torch.equal(fields[0], fields[1]) and torch.equal(fields[0], fields[2])
    pad = [0.0] * (3 - len(n))
    so = oracle.setup(oracle.params(nharm=nharm, seed=seed, nc=nc + pad, fc=fc + pad, **kw))
    p = sb.make_params(nharm=nharm, seed=seed, nc=nc, fc=fc, **kw)
    tab, _, _ = sb.sample_device(p, sb.compute_setup(p))
    ref = gpu_fp64.structured_field(so, [1] * 3, list(n) + [1] * (3 - len(n)), ds, tab)
    err = float((fields[0].double() - ref).square().mean().sqrt() / ref.square().mean().sqrt())
    assert err <= tol, err
