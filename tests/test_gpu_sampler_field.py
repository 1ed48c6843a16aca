"""The single-field form of the device sampler against the serial host loop, bit
for bit: one block and many, one chunk per block and several (where it also
takes the certain-reject thresholds), every harmonic kept and some above the
cut, negative and zero seeds, 2-D and 3-D spectra; repeated calls and two
threads at once."""
import threading

import numpy as np
import pytest

import scarf3d_b200 as sb

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _params(acf=0, nd=3, cl=600.0, nharm=700, seed=9, ds=50.0, dh=None, span=6000.0):
    return sb.make_params(acf=acf, nharm=nharm, seed=seed, hurst=0.4 if acf == 0 else 0.0, sigma=0.05, ds=ds, dh=dh,
                          cl=[cl] * nd, nc=[0.0] * 3, fc=[span] * nd + [0.0] * (3 - nd))


def _same(p):
    s = sb.compute_setup(p)
    tab, used, _ = sb.sample_device(p, s)
    ref, ref_used = sb.sample(p, s)
    assert used == ref_used and np.array_equal(tab.view(np.uint32), ref.view(np.uint32))


@pytest.mark.parametrize("kw", [
    dict(nharm=1), dict(nharm=2, seed=0), dict(nharm=63, seed=-7), dict(nharm=20000, seed=123456789),
    dict(acf=1), dict(acf=1, nd=2, cl=900.0, nharm=3001), dict(nd=2, nharm=501),
    dict(ds=400.0, dh=50.0, nharm=4000),              # harmonics above the cut are dropped
    dict(acf=1, cl=2600.0, span=6000.0, nharm=4000),  # rare acceptance: several chunks per block
])
def test_tables_match_the_host_loop(kw):
    _same(_params(**kw))


def test_repeated_and_threaded_calls():
    ps = [_params(nharm=900 + 300 * i, seed=i) for i in range(4)]
    ss = [sb.compute_setup(p) for p in ps]
    ref = [sb.sample(p, s)[0] for p, s in zip(ps, ss)]
    bad = []

    def work(i):
        for _ in range(5):
            if not np.array_equal(sb.sample_device(ps[i], ss[i])[0].view(np.uint32), ref[i].view(np.uint32)):
                bad.append(i)

    ths = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in ths:
        t.start()
    for t in ths:
        t.join()
    assert not bad
