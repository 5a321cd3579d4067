"""Rotor-model annealing on both sides of the sample counts above which one
thread takes a sample, against the oracle bit for bit: every proposal and order,
repeated couplers and self-loops, schedules at the ends of the number range."""
import numpy as np
import pytest

import oracle
from b200sa.sqa import simulated_annealing
from conftest import bits

pytestmark = pytest.mark.gpu


def line(proposal, order, n):
    if "NonErgodic" in proposal:
        if n > 128:
            return None
        if not order:
            return 4096 if n <= 16 else 256 * n
        return 2560 if n <= 32 else 80 * n if n <= 64 else 32768
    if not order:
        return 4096 + 16 * n
    return 2560 if n <= 53 else 48 * n if n <= 256 else 64 * n


def check(n, R, proposal, order, hp, hd, spb=1):
    rng = np.random.default_rng(n + R)
    u, v = (rng.integers(0, n, 2 * n).astype(np.int32) for _ in range(2))
    J, h, tf = rng.normal(0, 1, 2 * n), rng.normal(0, 0.3, n), rng.uniform(0, 2, n)
    st0 = rng.integers(0, 256, (R, n)).astype(np.uint8)
    with np.errstate(all="ignore"):
        ws, we, wst = oracle.rotormc(h, u, v, J, tf, st0, spb, hp, hd, 91 + np.arange(R), order, proposal, 2)
        s, e, st = simulated_annealing(R, h, u, v, J, tf, spb, hp, hd, 91, st0.copy(), order, proposal, 2)
    np.testing.assert_array_equal(s, ws)
    np.testing.assert_array_equal(bits(e), bits(we))
    np.testing.assert_array_equal(st, wst)


@pytest.mark.parametrize("proposal", list(oracle.ROTOR_PROPOSALS))
@pytest.mark.parametrize("order", [False, True])
@pytest.mark.parametrize("n", [1, 9, 16, 33, 64, 128, 129])
def test_both_sides_of_the_line(n, order, proposal):
    R = line(proposal, order, n)
    hp, hd = np.geomspace(0.1, 20.0, 3), np.geomspace(10.0, 0.01, 3)
    for k in ([40000] if R is None else [R, R + 1]):
        check(n, k, proposal, order, hp, hd)


@pytest.mark.parametrize("proposal", list(oracle.ROTOR_PROPOSALS))
@pytest.mark.parametrize("order", [False, True])
def test_schedule_extremes(order, proposal):
    check(12, 5001, proposal, order, np.array([1e-300, 1.0, 1e300, 0.0, -1.0]),
          np.array([1.0, 1e-9, 1.0, 0.5, 0.25]), spb=2)
