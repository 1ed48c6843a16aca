"""The single-field sampler where the pairs of its first scan run out: few
harmonics of a rare acceptance, many seeds (about one in six runs out), against
the serial host loop bit for bit, with the same number of pairs used."""
import numpy as np
import pytest

import scarf3d_b200 as sb

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("acf,cl,nharm", [(0, 4000.0, 100), (0, 5000.0, 100), (1, 4000.0, 20), (1, 2600.0, 37),
                                          (0, 4000.0, 1)])
def test_tables_match_the_host_loop(acf, cl, nharm):
    for seed in range(1, 25):
        p = sb.make_params(acf=acf, nharm=nharm, seed=seed, hurst=0.4 if acf == 0 else 0.0, sigma=0.05, ds=50.0,
                           cl=[cl] * 3, nc=[0.0] * 3, fc=[6000.0] * 3)
        s = sb.compute_setup(p)
        tab, used, _ = sb.sample_device(p, s)
        ref, ref_used = sb.sample(p, s)
        assert used == ref_used and np.array_equal(tab.view(np.uint32), ref.view(np.uint32))
