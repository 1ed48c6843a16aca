"""The FIM's inverse transform over axis lengths of its forms (plain, and
Rader's or Bluestein's for prime factors above 5), even and odd half lengths, tiles that the
x bins and rows do not fill, two-point axes, and axes beyond shared memory
(cuFFT), through scarf_execute against the FP64 transform of the oracle.

Tolerance: FP32 transforms of at most ~1 100 points, three axes of up to two
transforms with ~11 levels each and ~6e-8 a level, a few 1e-7 in all; 2e-6."""
import numpy as np
import pytest

import scarf3d_b200 as sb
from conftest import rel_rms
from oracle import fim

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

DS = 50.0


def _run(internal, acf=0, **kw):
    """A field whose internal grid has the given (even) axis lengths."""
    nd = len(internal)
    fe = [n - 1 for n in internal]
    cl = [max(0.1 * n * DS, 2.5 * DS) for n in internal]
    par = dict(ds=DS, acf=acf, cl=cl, sigma=0.05, hurst=0.4 if acf == 0 else 0.0, pad=0, **kw)
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


@pytest.mark.parametrize("internal", [
    (48, 40, 36), (46, 58, 62), (8, 14, 22), (34, 4, 6), (4, 2, 26), (130, 50, 34), (258, 30, 24), (16, 514, 10),
    (30, 8, 514)])
def test_three_dimensions(internal):
    _run(internal)


@pytest.mark.parametrize("internal", [(514, 78), (64, 96), (94, 1028), (1026, 34), (1902, 50), (50, 1902)])
def test_two_dimensions(internal):
    _run(internal, acf=1)


def test_rescaled():
    _run((38, 46, 30), rescale=1)


@pytest.mark.parametrize("internal", [
    # y and z: q = 2 to 54 blocks, p - 1 as one butterfly (7, 11, 13) and as
    # several stages, one and more q-point stages; x: the halves 7 (too short for
    # a plan of two stages), 17, 19, 31 (one block), 14, 28, 65, 257 and 541
    (14, 22, 26), (34, 14, 84), (38, 66, 52), (62, 100, 34), (28, 140, 22), (56, 38, 76), (130, 202, 14),
    (514, 26, 82), (1082, 8, 14)])
def test_rader_form(internal):
    _run(internal)


@pytest.mark.parametrize("internal", [(44, 1026), (1538, 38), (26, 1082), (102, 420), (36, 462)])
def test_rader_form_long(internal):
    # 54 blocks of 19, halves of 769, two blocks of 541, 60 blocks of 7; 462 = 6 x 7 x 11 has two primes (Bluestein)
    _run(internal)


@pytest.mark.parametrize("internal", [
    # radix 7: plain lengths (halves of 49, 35 and 21), p - 1 with a factor 7 (29, 43, 71, 113), 7 in q
    (98, 42, 28), (70, 126, 14), (42, 58, 86), (58, 98, 142), (172, 28, 226), (154, 34, 20), (258, 14, 258)])
def test_factors_of_seven(internal):
    _run(internal)
