"""The phases of the FIM's spectrum are the reference's: the single-precision
product of the draw, 2 and pi (scarflib_fim.f90's h), not the exact 2 pi u, from
which it differs by up to 2.4e-7. Both choices are transformed in FP64; the field
has to lie nearer to the reference's."""
import numpy as np
import pytest

import oracle
import scarf3d_b200 as sb
from oracle import fim

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

DS, SEED = 50.0, 31


@pytest.mark.parametrize("n,acf", [((63, 63), 1), ((47, 39, 35), 0), ((40, 47, 38), 1)])
def test_phases_are_rounded_as_the_references(n, acf, monkeypatch):
    nd = len(n)
    par = dict(ds=DS, acf=acf, cl=[max(0.1 * v * DS, 125.0) for v in n], sigma=0.05, hurst=0.4 if acf == 0 else 0.0)
    try:
        sb.scarf_initialize(fs=[1] * nd, fe=list(n), method=0, **par)
        got = sb.scarf_execute(SEED, torch.empty(int(np.prod(n)), device="cuda"))[0].cpu().numpy().astype(np.float64)
    finally:
        sb.scarf_finalize()
    case = dict(fs=[1] * nd, fe=list(n), seed=SEED, **par)
    ref = fim.execute_structured(**case)[0]
    spectrum = fim.spectrum

    def exact_phases(npts, *args):
        # turns every inner bin (the Hermitian planes keep theirs) from the
        # rounded phase to the exact one
        n1, n2, n3 = npts
        u = (oracle.raw_stream(SEED, n1 * n2 * n3).astype(np.float64) * float.fromhex("0x1.00000002p-31"))
        u = u.astype(np.float32).reshape(n3, n2, n1)[..., :n1 // 2 + 1]
        h = (u * np.float32(2.0)) * np.float32(np.pi)
        turn = np.exp(1j * (2.0 * np.pi * u.astype(np.float64) - h.astype(np.float64)))
        turn[..., 0] = turn[..., -1] = 1.0
        return spectrum(npts, *args) * turn

    monkeypatch.setattr(fim, "spectrum", exact_phases)
    other = fim.execute_structured(**case)[0]
    near, far = (float(np.sqrt(np.mean((got - r) ** 2))) for r in (ref, other))
    assert near < far, (near / ref.std(), far / ref.std())
