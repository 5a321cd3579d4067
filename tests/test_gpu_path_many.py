"""Path-integral annealing around the number of samples from which a thread
serves a sample: the samples of the larger call are those of the smaller one,
and the last ones equal the oracle's."""
import numpy as np
import pytest

import oracle
from conftest import bits
from test_gpu_path_warps import run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(3, 4), (5, 10)])
def test_around_the_rule(n, m):
    hd, hp, most = [3.0, 0.5], [0.5, 2.0], 40960
    h, u, v, J, s0, _, _, _, _, st, en, nb, out = run(n, m, most + 33, hd, hp)
    # run() draws the problem before the states: the smaller call has the same ones.
    small = run(n, m, most, hd, hp)
    np.testing.assert_array_equal(st[:most], small[9])
    np.testing.assert_array_equal(bits(en[:most]), bits(small[10]))
    np.testing.assert_array_equal(nb[:most], small[11])
    total = nb[:most].sum()
    np.testing.assert_array_equal(out[:total], small[12][:total])
    for r in range(most, most + 33):
        ws, we, _, wnb, _ = oracle.pimc(h, u, v, J, s0[r:r + 1], 1, hp, hd, 5 + r, 0.0, 1, 1, True, False,
                                        max_out=256)
        np.testing.assert_array_equal(st[r:r + 1], ws)
        np.testing.assert_array_equal(bits(en[r:r + 1]), bits(we))
        np.testing.assert_array_equal(nb[r:r + 1], wnb)
