"""Path-integral annealing on both sides of the sample count from which a thread
serves a sample, for fields and degrees that move it: the samples of the larger
call are those of the smaller one, and every 50th equals the oracle's."""
import numpy as np
import pytest

import oracle
from conftest import bits
from test_gpu_path_warps import run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,hd", [(1, 0, [0.2, 0.05]), (6, 0, [0.0, 0.0]), (9, 9, [0.4, 0.1]), (20, 90, [0.5, 0.1]),
                                    (40, 40, [1.0, 0.2])])
def test_both_sides_of_the_line(n, m, hd):
    line = int(4350 * (1 + 2.65 * np.mean(hd)) * (1 + m / n / 6) * n ** (1 / 6))
    assert 4350 <= line < 40960
    hp = [0.5, 2.0]
    h, u, v, J, s0, _, _, _, _, st, en, nb, out = run(n, m, line + 40, hd, hp)
    small = run(n, m, line - 1, hd, hp)
    r = line - 1
    np.testing.assert_array_equal(st[:r], small[9])
    np.testing.assert_array_equal(bits(en[:r]), bits(small[10]))
    np.testing.assert_array_equal(nb[:r], small[11])
    total = nb[:r].sum()
    np.testing.assert_array_equal(out[:total], small[12][:total])
    for r in range(0, line + 40, 50):
        ws, we, _, wnb, _ = oracle.pimc(h, u, v, J, s0[r:r + 1], 1, hp, hd, 5 + r, 0.0, 1, 1, True, False,
                                        max_out=256)
        np.testing.assert_array_equal(st[r:r + 1], ws)
        np.testing.assert_array_equal(bits(en[r:r + 1]), bits(we))
        np.testing.assert_array_equal(nb[r:r + 1], wnb)
