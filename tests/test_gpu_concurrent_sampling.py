"""scarf_execute beside the sampling entry points in other threads, which share
the device sampler's buffers with it: every field and every table is bit for
bit that of the same call made alone."""
import threading

import numpy as np
import pytest

import scarf3d_b200 as sb

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _params(nharm, seed):
    return sb.make_params(acf=0, nharm=nharm, seed=seed, hurst=0.4, sigma=0.05, ds=50.0, cl=[600.0] * 3,
                          nc=[0.0] * 3, fc=[6000.0] * 3)


# harmonics of the other threads' tables: below, above and far above the
# field's, so that the sampler's buffers are rewritten and reallocated
@pytest.mark.parametrize("others", [(500, 4000), (200, 60000, 9000)])
@pytest.mark.parametrize("form", [sb.FORM_AUTO, sb.FORM_DIRECT])
def test_fields_beside_other_threads_tables(others, form):
    sb.release_device_memory()
    ps = [_params(n, 31 + n) for n in others]
    ss = [sb.compute_setup(p) for p in ps]
    refs = [sb.sample(p, s)[0] for p, s in zip(ps, ss)]
    sb.set_nharm(3000)
    sb.set_form(form)
    stop, wrong = threading.Event(), []

    def tables():
        while not stop.is_set():
            for p, s, ref in zip(ps, ss, refs):
                if not np.array_equal(sb.sample_device(p, s)[0].view(np.uint32), ref.view(np.uint32)):
                    wrong.append(p.nharm)

    try:
        sb.scarf_initialize(fs=[1] * 3, fe=[64, 48, 40], ds=50.0, acf=0, cl=[300.0] * 3, sigma=0.05, hurst=0.3,
                            method=1)
        seeds = range(1, 13)
        alone = [sb.scarf_execute(seed, torch.zeros(64 * 48 * 40, device="cuda"))[0] for seed in seeds]
        ths = [threading.Thread(target=tables) for _ in range(2)]
        for t in ths:
            t.start()
        try:
            for _ in range(4):
                for seed, ref in zip(seeds, alone):
                    field, _ = sb.scarf_execute(seed, torch.zeros(64 * 48 * 40, device="cuda"))
                    if not torch.equal(field, ref):
                        wrong.append(-seed)
        finally:
            stop.set()
            for t in ths:
                t.join()
    finally:
        sb.scarf_finalize()
        sb.set_nharm(10000)
        sb.set_form(sb.FORM_AUTO)
    assert not wrong
