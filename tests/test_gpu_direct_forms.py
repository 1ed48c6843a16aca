"""The two forms of the FP32 direct sum (packed pairs of points per thread for
large sets, ordered terms for small ones) give the same field bit for bit: each
point adds its harmonics in table order in both. Sizes at the edges of blocks,
harmonic tiles and batches; the small sets also against the CPU restatement
of the reference's FP32 sum, at the tolerance of that comparison elsewhere
(1e-6: the sines and cosines differ by ulps)."""
import ctypes

import numpy as np
import pytest

import oracle
import scarf3d_b200 as sb
from conftest import rel_rms
from srm_cases import random_points

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

KW = dict(acf=1, seed=7, hurst=0.0, sigma=0.1, ds=100.0, cl=[1500.0, 1500.0, 500.0])
BOX = dict(nc=[0.0, 0.0, 0.0], fc=[20000.0, 20000.0, 10000.0])


def _sum(s, xyz, tab):
    n = len(xyz[0])
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (*xyz, tab.reshape(-1))]
    out = torch.full((n,), float("nan"), device="cuda")
    sb.check(sb.lib.scarf_srm_direct_points(ctypes.byref(s), *(ctypes.c_void_p(a.data_ptr()) for a in d[:3]), n,
                                            ctypes.c_void_p(d[3].data_ptr()), len(tab),
                                            ctypes.c_void_p(out.data_ptr()), None))
    return out.cpu().numpy()


@pytest.mark.parametrize("mode,large", [(sb.SINCOS_FAST, 60001 + 255), (sb.SINCOS_ACCURATE, 100001)])
@pytest.mark.parametrize("nharm", [1, 2, 63, 64, 65, 127, 128, 129, 700])
def test_forms_agree_bit_for_bit(mode, large, nharm):
    p = sb.make_params(nharm=nharm, **KW, **BOX)
    s = sb.compute_setup(p)
    tab, _ = sb.sample(p, s)
    xyz = random_points(large, seed=3)
    try:
        sb.set_direct_sincos(mode)
        packed = _sum(s, xyz, tab)
        for n in (1, 31, 32, 33, 1000):
            ordered = _sum(s, [a[:n] for a in xyz], tab)
            assert np.array_equal(ordered.view(np.uint32), packed[:n].view(np.uint32)), n
    finally:
        sb.set_direct_sincos(sb.SINCOS_FAST)
    so = oracle.setup(oracle.params(nharm=nharm, **KW, **BOX))
    ref = oracle.sum_points(so, *[a[:1000] for a in xyz], tab)
    assert rel_rms(packed[:1000], ref) <= 1e-6
