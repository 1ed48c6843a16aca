"""The FIM on grids whose long axis takes cuFFT, where the scaling of the
transform is left to the step that reads the internal field next: with rescale,
with a taper, with both and into a host array, against the oracle.

Tolerance: FP32 transforms of ~1 900 points, a few 1e-7; 2e-6 as for the other
lengths, 3e-6 with rescale, whose division by the FP32 deviation adds roundings."""
import numpy as np
import pytest

import scarf3d_b200 as sb
from conftest import rel_rms
from oracle import fim

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

DS = 50.0
# 1902 = 6 x 317: Bluestein's form of it exceeds shared memory
GRIDS = [(50, 1902), (6, 8, 1902)]
POI = dict(mute=400.0, taper=1500.0)


@pytest.mark.parametrize("internal", GRIDS)
@pytest.mark.parametrize("kw,host", [({}, False), (dict(rescale=1), False), (dict(poi=1, **POI), False),
                                     (dict(rescale=1, poi=1, **POI), False), (dict(rescale=1, poi=1, **POI), True)])
def test_scaling_is_applied_once(internal, kw, host):
    nd = len(internal)
    fe = [n - 1 for n in internal]
    kw = dict(kw)
    if "poi" in kw:
        kw["poi"] = np.array([[0.3 * n * DS for n in fe]], np.float32)
    cl = [max(0.1 * n * DS, 2.5 * DS) for n in internal]
    par = dict(ds=DS, acf=0, cl=cl, sigma=0.05, hurst=0.4, pad=0, **kw)
    assert sb.fim_internal_grid(nd, [0.0] * nd, [(f - 1) * DS for f in fe], DS, cl)[0][:nd] == list(internal)
    npts = int(np.prod(fe))
    try:
        sb.scarf_initialize(fs=[1] * nd, fe=fe, method=0, **par)
        field = np.full(npts, np.nan, np.float32) if host else torch.full((npts,), float("nan"), device="cuda")
        _, stats = sb.scarf_execute(31, field)
    finally:
        sb.scarf_finalize()
    ref, info, _ = fim.execute_structured(fs=[1] * nd, fe=fe, seed=31, **par)
    got = field if host else field.cpu().numpy()
    tol = 3e-6 if "rescale" in kw else 2e-6
    assert rel_rms(got, ref) <= tol, rel_rms(got, ref)
    assert abs(stats[2] / info[2] - 1) <= 1e-5 and abs(stats[3] - info[3]) <= 1e-5 * info[2]
