"""Planning of the FIM's transforms on the host, part of every execute: grids
whose axes need a search for a convolution length (large prime factors) cost
little, and their plans (by the workspace, which holds the tables of the
convolution's length) are the ones an exhaustive search finds."""
import ctypes
import time

import pytest

import scarf3d_b200 as sb

GRIDS = [((66, 66, 1), 39424), ((514, 514, 514), 1089314560), ((1002, 1002, 1), 8107520),
         ((1702, 1702, 1), 23300608), ((402, 3502, 1), 11299328), ((50, 1702, 50), 35047424),
         ((3002, 3002, 1), 72148992), ((80, 1409, 1), 976640), ((566, 1433, 1), 6575360)]


@pytest.mark.parametrize("npts,nbytes", GRIDS)
def test_plans_are_found_quickly(npts, nbytes):
    f = sb.lib.scarf_fim_workspace_bytes
    a, best = (ctypes.c_int * 3)(*npts), 1.0
    for _ in range(200):
        t = time.perf_counter()
        got = f(a, 0)
        best = min(best, time.perf_counter() - t)
        assert got == nbytes
    # 4 to 8 us; trying every length and factorisation took 21 to 57
    assert best < 15e-6
