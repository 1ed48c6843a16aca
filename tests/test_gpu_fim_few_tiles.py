"""The FIM's transforms where their tiles are few or large, for which a block
takes more threads than the usual 256: long axes beside short ones, of each form
(plain, Rader's, Bluestein's), along each axis, against the FP64 transform of
the oracle.

Tolerance: at most ~3 500 points and two transforms an axis, 24 levels of
~6e-8 each in a random walk over three axes, 5e-7; 2e-6."""
import numpy as np
import pytest

import scarf3d_b200 as sb
from conftest import rel_rms
from oracle import fim

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

DS = 50.0


@pytest.mark.parametrize("internal", [
    (80, 1410), (568, 1434), (14, 934), (4, 1410), (50, 1702, 10), (8, 6, 794), (6, 1786), (1702, 8), (3406, 6),
    (4, 2048), (6, 3500), (4096, 4), (300, 1024), (4, 1538), (1538, 4), (8, 4, 1082), (514, 8, 6)])
@pytest.mark.parametrize("kw", [{}, {"rescale": 1}])
def test_long_axes(internal, kw):
    nd = len(internal)
    fe = [n - 1 for n in internal]
    cl = [max(0.1 * n * DS, 2.5 * DS) for n in internal]
    par = dict(ds=DS, acf=0, cl=cl, sigma=0.05, hurst=0.4, pad=0, **kw)
    assert sb.fim_internal_grid(nd, [0.0] * nd, [(f - 1) * DS for f in fe], DS, cl)[0][:nd] == list(internal)
    try:
        sb.scarf_initialize(fs=[1] * nd, fe=fe, method=0, **par)
        dev = torch.full((int(np.prod(fe)),), float("nan"), device="cuda")
        _, stats = sb.scarf_execute(31, dev)
    finally:
        sb.scarf_finalize()
    ref, info, _ = fim.execute_structured(fs=[1] * nd, fe=fe, seed=31, **par)
    got = dev.cpu().numpy()
    assert rel_rms(got, ref) <= 2e-6, rel_rms(got, ref)
    assert abs(stats[2] / info[2] - 1) <= 1e-5 and abs(stats[3] - info[3]) <= 1e-5 * info[2]
