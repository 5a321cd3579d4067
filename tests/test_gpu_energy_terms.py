"""The final energy's sum, 32 terms at a time: numbers of variables and couplers
around a multiple of 32, no couplers, lists long enough to be read in groups,
spins of any value, every state location and order.  Energies and spins equal
the oracle's."""
import numpy as np
import pytest

import oracle
from b200sa import simulated_annealing
from conftest import bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("random_order", [False, True])
@pytest.mark.parametrize("n,m", [(352, 0), (353, 1), (351, 31), (352, 32), (353, 33), (383, 64), (352, 4095),
                                 (1500, 9000), (5000, 12001)])
def test_energy(n, m, random_order):
    rng = np.random.default_rng(n + m)
    key = rng.permutation(n * (n - 1))[:m]
    u = (key // (n - 1)).astype(np.int32)
    v = (key % (n - 1)).astype(np.int32)
    v += v >= u
    J, h = rng.normal(0, 1, m), rng.normal(0, 1, n)
    s0 = (2 * rng.integers(0, 2, (6, n)) - 1).astype(np.int8)
    s0[4:] = rng.integers(-3, 4, (2, n))
    betas = np.array([0.3, 2.0])
    ws, we = oracle.run(h, u, v, J, s0, 1, betas, (7 + np.arange(6)).astype(np.uint64), random_order)
    s, e = simulated_annealing(6, h, u, v, J, 1, betas, 7, s0.copy(), random_order)
    np.testing.assert_array_equal(s, ws)
    np.testing.assert_array_equal(bits(e), bits(we))
