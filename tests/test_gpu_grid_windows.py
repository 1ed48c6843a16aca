"""The gridded sum where the harmonics' z factors do not fit their bounded buffer
for all planes at once: they are built several times, for the planes of one pass
after another (the last one partial), in the places that the first build found.
Against the FP64 sum over the same harmonics, and the workspace stays bounded.

Tolerance: that of tests/test_gpu_grid_dense_bins.py for 300 000 harmonics."""
import numpy as np
import pytest

import oracle
import scarf3d_b200 as sb
from oracle import gpu_fp64

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,frac", [((24, 20, 330), 0.05), ((24, 20, 330), 0.4), ((24, 700), 0.05), ((40, 1100), 0.4)])
def test_factors_built_in_several_windows(n, frac):
    ds, seed, nharm = 25.0, 11, 300000
    span = max(n) * ds
    kw = dict(acf=0, hurst=0.4, sigma=0.05, ds=ds, cl=[frac * span] * len(n), alpha=20.0)
    nc, fc = [0.0] * len(n), [span] * len(n)
    sb.release_device_memory()
    sb.set_nharm(nharm)
    try:
        sb.scarf_initialize(fs=[1] * len(n), fe=list(n), method=1, nc=nc, fc=fc, **kw)
        field, _ = sb.scarf_execute(seed, torch.full((int(np.prod(n)),), float("nan"), device="cuda"))
        again, _ = sb.scarf_execute(seed, torch.full((int(np.prod(n)),), float("nan"), device="cuda"))
        # 2^30 bytes of factors, as much of partial sums at most, and the rest
        # (2 MB of harmonics' tables, grids of under 2 MB a plane)
        assert sb.device_memory_in_use() < 3 << 30
    finally:
        sb.scarf_finalize()
        sb.set_nharm(10000)
        sb.release_device_memory()
    assert torch.equal(field, again)
    pad = [0.0] * (3 - len(n))
    so = oracle.setup(oracle.params(nharm=nharm, seed=seed, nc=nc + pad, fc=fc + pad, **kw))
    p = sb.make_params(nharm=nharm, seed=seed, nc=nc, fc=fc, **kw)
    tab, _, _ = sb.sample_device(p, sb.compute_setup(p))
    ref = gpu_fp64.structured_field(so, [1] * 3, list(n) + [1] * (3 - len(n)), ds, tab)
    err = float((field.double() - ref).square().mean().sqrt() / ref.square().mean().sqrt())
    assert err <= 4e-6, err
