"""The gridded sum at its limits: under a device-memory cap it takes smaller
passes, then leaves the sum to the tensor-core form, with the right field each
time; and device fields that are only 4-byte aligned."""
import numpy as np
import pytest

import oracle
import scarf3d_b200 as sb
from oracle import gpu_fp64

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

N, DS, SEED = (160, 120, 200), 25.0, 7
KW = dict(acf=0, hurst=0.4, sigma=0.05, ds=DS, cl=[400.0] * 3)


@pytest.fixture(autouse=True)
def _reset():
    yield
    sb.scarf_finalize()
    sb.set_nharm(10000)
    sb.set_form(sb.FORM_AUTO)
    sb.set_device_memory_cap(0)
    sb.release_device_memory()


def _init(n=N, nharm=3000, method=1):
    sb.set_nharm(nharm)
    sb.scarf_initialize(fs=[1] * len(n), fe=list(n), method=method, **KW)


def _execute(form=sb.FORM_AUTO):
    sb.release_device_memory()
    sb.set_form(form)
    field, stats = sb.scarf_execute(SEED, torch.full((int(np.prod(N)),), float("nan"), device="cuda"))
    return field, stats[:4].copy(), sb.device_memory_in_use()


def test_memory_caps():
    _init()
    grid, grid_stats, most = _execute()
    tc, _, least = _execute(sb.FORM_TC)
    assert least < most and not torch.equal(grid, tc)
    so = oracle.setup(oracle.structured_params(nharm=3000, seed=SEED, fs=[1] * 3, fe=list(N), **KW))
    tab, _ = oracle.sample(oracle.structured_params(nharm=3000, seed=SEED, fs=[1] * 3, fe=list(N), **KW), so)
    ref = gpu_fp64.structured_field(so, [1] * 3, list(N), DS, tab)
    rms = ref.square().mean().sqrt()
    smaller, contracted = 0, 0
    for step in range(17):
        sb.set_device_memory_cap(int(most - (most - least) * step / 16))
        field, stats, used = _execute()
        err = float((field.double() - ref).square().mean().sqrt() / rms)
        if torch.equal(field, tc):
            contracted += 1
            assert err <= 1e-5, err
        else:
            smaller += used < most
            assert err <= 2e-6, err
            # the statistics of more, smaller records: FP64 sums in another order
            assert np.allclose(stats, grid_stats, rtol=1e-6, atol=1e-9)
    assert smaller > 0 and contracted > 0


@pytest.mark.parametrize("n", [(160, 120, 40), (161, 120, 40), (800, 300)])
@pytest.mark.parametrize("method,form", [(1, sb.FORM_AUTO), (1, sb.FORM_TC), (1, sb.FORM_DIRECT), (0, sb.FORM_AUTO)])
def test_fields_of_four_byte_alignment(n, method, form):
    kw = dict(KW, cl=[400.0] * len(n))
    sb.set_nharm(3000)
    sb.set_form(form)
    sb.scarf_initialize(fs=[1] * len(n), fe=list(n), method=method, **kw)
    npts = int(np.prod(n))
    whole, stats = sb.scarf_execute(SEED, torch.full((npts,), float("nan"), device="cuda"))
    room = torch.full((npts + 2,), float("nan"), device="cuda")
    odd = room[1:npts + 1]
    assert odd.data_ptr() % 8 == 4
    _, odd_stats = sb.scarf_execute(SEED, odd)
    assert torch.equal(odd, whole) and np.allclose(stats[:4], odd_stats[:4], rtol=1e-6, atol=1e-9)
    assert torch.isnan(room[0]) and torch.isnan(room[-1])
