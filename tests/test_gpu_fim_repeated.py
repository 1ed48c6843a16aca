"""The tables of the FIM's transforms, which stay with a context for the next
call on the same internal grid: grids that take turns, with sums by the other
method (which use the same workspace) and the release of the library's buffers
between, give the field that a fresh context gives, bit for bit."""
import numpy as np
import pytest

import scarf3d_b200 as sb

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# transforms of each form, tables of equal and different sizes, a grid whose
# long axis takes cuFFT, two and three dimensions
GRIDS = [(46, 38, 34), (44, 56, 60), (512, 76), (76, 512), (48, 1900), (61, 61, 61), (60, 62, 61)]


def _init(n, method=0):
    sb.scarf_initialize(fs=[1] * len(n), fe=list(n), ds=50.0, acf=0, cl=[max(0.1 * v * 50.0, 125.0) for v in n],
                        sigma=0.05, hurst=0.3, method=method)


def _field(n, seed):
    dev, stats = sb.scarf_execute(seed, torch.full((int(np.prod(n)),), float("nan"), device="cuda"))
    return dev, stats[:4].copy()


def _fresh(n, seed):
    c = sb.Context()
    try:
        with c:
            _init(n)
            out = _field(n, seed)
            sb.scarf_finalize()
        return out
    finally:
        c.close()


def test_grids_take_turns():
    ref = {n: [_fresh(n, seed) for seed in (1, 2)] for n in GRIDS}
    sb.set_nharm(2000)
    try:
        for between in ("nothing", "sum", "release"):
            for n in GRIDS + GRIDS[::-1]:
                _init(n)
                for _ in range(2):
                    for seed in (1, 2):
                        dev, stats = _field(n, seed)
                        assert torch.equal(dev, ref[n][seed - 1][0]), (between, n)
                        assert np.array_equal(stats, ref[n][seed - 1][1]), (between, n)
                    if between == "sum":
                        sb.scarf_finalize()
                        _init((64, 48, 40), method=1)
                        _field((64, 48, 40), 3)
                        sb.scarf_finalize()
                        _init(n)
                    elif between == "release":
                        sb.release_device_memory()
                sb.scarf_finalize()
    finally:
        sb.scarf_finalize()
        sb.set_nharm(10000)
