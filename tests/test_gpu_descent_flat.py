"""Steepest descent that looks at every variable in each step: both sides of
the line between it and group minima, equal energies, repeated couplers, state
in shared memory and in global slots; every result equals the oracle's."""
import numpy as np
import pytest

import oracle
from b200sa.greedy import steepest_gradient_descent
from conftest import bits

pytestmark = pytest.mark.gpu


def check(h, u, v, J, s0, sparse):
    ws, we, wk = oracle.descent(h, u, v, J, s0, sparse)
    s, e, k = steepest_gradient_descent(len(s0), h, u, v, J, s0.copy(), sparse)
    np.testing.assert_array_equal(s, ws)
    np.testing.assert_array_equal(bits(e), bits(we))
    np.testing.assert_array_equal(k, wk)


@pytest.mark.parametrize("sparse", [False, True])
@pytest.mark.parametrize("weights", ["integer", "normal"])
@pytest.mark.parametrize("n,m", [(255, 300), (256, 300), (257, 300), (300, 3749), (300, 3750), (300, 44850), (600, 90000)])
def test_steps_that_look_at_every_variable(n, m, weights, sparse):
    """Both sides of the line: 256 variables, 24 m = n^2."""
    rng = np.random.default_rng(n + m)
    u, v = np.triu_indices(n, 1)
    keep = np.sort(rng.choice(u.size, m, replace=False))
    u, v = u[keep].astype(np.int32), v[keep].astype(np.int32)
    integer = weights == "integer"
    J = rng.integers(-2, 3, m).astype(float) if integer else rng.normal(0, 1, m)
    h = rng.integers(-1, 2, n).astype(float) if integer else rng.normal(0, 0.3, n)
    s0 = (2 * rng.integers(0, 2, (6, n)) - 1).astype(np.int8)
    check(h, u, v, J, s0, sparse)


@pytest.mark.parametrize("sparse", [False, True])
def test_every_variable_in_global_slots(sparse):
    """Too few warps fit on chip for so many samples: each starts three flips from
    a minimum."""
    rng = np.random.default_rng(4)
    n, m, R = 2500, 262000, 2700
    u, v = rng.integers(0, n, m).astype(np.int32), rng.integers(0, n, m).astype(np.int32)
    u, v = u[u != v], v[u != v]
    J, h = rng.normal(0, 1, u.size), rng.normal(0, 1, n)
    low = oracle.descent(h, u, v, J, (2 * rng.integers(0, 2, (1, n)) - 1).astype(np.int8), sparse)[0]
    s0 = np.repeat(low, R, axis=0)
    s0[np.arange(R)[:, None], rng.integers(0, n, (R, 3))] *= -1
    check(h, u, v, J, s0, sparse)
