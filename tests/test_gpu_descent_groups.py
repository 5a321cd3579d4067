"""Steepest descent with minima kept per group of 32 variables: sizes around a
group and around 32 groups, equal energies (ties to the lowest index), lists
longer than a warp, repeated couplers, state in shared memory and in global
slots; every result equals the oracle's."""
import numpy as np
import pytest

import oracle
from b200sa.greedy import steepest_gradient_descent
from conftest import bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sparse", [False, True])
@pytest.mark.parametrize("weights", ["integer", "normal"])
@pytest.mark.parametrize("n,m,R", [(1, 0, 3), (2, 1, 4), (31, 200, 9), (32, 90, 9), (33, 60, 9), (64, 2000, 7),
                                   (1023, 3000, 9), (1025, 2000, 9), (2100, 40000, 5), (8200, 9000, 4),
                                   (20000, 60000, 2)])
def test_groups(n, m, R, weights, sparse):
    rng = np.random.default_rng(n)
    u, v = (rng.integers(0, n, m).astype(np.int32) for _ in range(2))
    u, v = u[u != v], v[u != v]
    integer = weights == "integer"  # small integers: many equal flip energies
    J = rng.integers(-2, 3, len(u)).astype(float) if integer else rng.normal(0, 1, len(u))
    h = rng.integers(-1, 2, n).astype(float) if integer else rng.normal(0, 0.3, n)
    s0 = (2 * rng.integers(0, 2, (R, n)) - 1).astype(np.int8)
    ws, we, wk = oracle.descent(h, u, v, J, s0, sparse)
    s, e, k = steepest_gradient_descent(R, h, u, v, J, s0.copy(), sparse)
    np.testing.assert_array_equal(s, ws)
    np.testing.assert_array_equal(bits(e), bits(we))
    np.testing.assert_array_equal(k, wk)
