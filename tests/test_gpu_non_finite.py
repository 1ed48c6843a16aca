"""Sums whose rotation or draws are not finite: every summation form gives a
field (and a mean) that are not numbers, as the reference's sum over such a
harmonic does, and the next call is unharmed."""
import ctypes

import numpy as np
import pytest

import oracle
import scarf3d_b200 as sb

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# 3-D and 2-D, and transform lengths with and without a last, partial bin
GRIDS = [(96, 80, 64), (250, 128, 33), (300, 288, 20), (640, 300), (37, 801)]
FORMS = [sb.FORM_AUTO, sb.FORM_TC, sb.FORM_DIRECT]


@pytest.fixture(autouse=True)
def _reset():
    yield
    sb.check(sb.lib.scarf_set_uniform_source(None, None))
    sb.scarf_finalize()
    sb.set_nharm(10000)
    sb.set_form(sb.FORM_AUTO)


def _init(n, alpha=0.0):
    sb.scarf_initialize(fs=[1] * len(n), fe=list(n), ds=25.0, acf=0, cl=[300.0] * len(n), sigma=0.05, hurst=0.3,
                        method=1, alpha=alpha)


def _execute(n):
    field, stats = sb.scarf_execute(5, torch.zeros(int(np.prod(n)), device="cuda"))
    return field.cpu().numpy(), stats


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("n", GRIDS)
def test_rotation_by_no_number(n, form):
    sb.set_nharm(3000)
    sb.set_form(form)
    _init(n)
    before, _ = _execute(n)
    sb.scarf_finalize()
    _init(n, alpha=float("nan"))
    field, stats = _execute(n)
    assert np.isnan(field).all() and np.isnan(stats[3])
    sb.scarf_finalize()
    _init(n)
    after, _ = _execute(n)
    assert np.isfinite(before).all() and np.array_equal(before, after)


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("n", GRIDS[:2] + GRIDS[3:4])
def test_draws_outside_the_unit_interval(n, form):
    # A source whose draws now and then leave [0, 1): arc cosines and square
    # roots of such draws are not numbers.
    state = (ctypes.c_int64 * 2)()
    count = [0]

    @ctypes.CFUNCTYPE(None, ctypes.c_int)
    def set_seed(seed):
        count[0] = 0
        oracle.L.orc_rng_seed(state, seed)

    @ctypes.CFUNCTYPE(None, ctypes.POINTER(ctypes.c_float))
    def srng(out):
        count[0] += 1
        out[0] = oracle.L.orc_u01(oracle.L.orc_rng_next(state))
        out[1] = oracle.L.orc_u01(oracle.L.orc_rng_next(state))
        if count[0] % 50 == 0:
            out[0], out[1] = 1.5, 1.5

    sb.set_nharm(3000)
    sb.set_form(form)
    sb.check(sb.lib.scarf_set_uniform_source(ctypes.cast(set_seed, ctypes.c_void_p),
                                             ctypes.cast(srng, ctypes.c_void_p)))
    _init(n)
    field, stats = _execute(n)
    assert np.isnan(field).all() and np.isnan(stats[3])
