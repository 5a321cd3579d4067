"""Calls of one sampler from two threads at once, of sizes whose launches differ
in shared memory by a factor of ten and more: each returns what it returns
alone."""
import threading

import numpy as np
import pytest

from b200sa import simulated_annealing, workloads
from b200sa.greedy import steepest_gradient_descent
from b200sa.sqa import path_annealing
from b200sa.sqa import simulated_annealing as rotor_annealing

pytestmark = pytest.mark.gpu


def anneal(n):
    rng, h, u, v, J = problem(n)
    return simulated_annealing(1, h, u, v, J, 1, [1.0], 3, workloads.random_states(rng, 1, n))


def descent(n):
    rng, h, u, v, J = problem(n)
    return steepest_gradient_descent(1, h, u, v, J, workloads.random_states(rng, 1, n))


def rotor(n):
    rng, h, u, v, J = problem(n)
    return rotor_annealing(1, h, u, v, J, np.ones(n), 1, [1.0], [0.5], 3,
                           rng.integers(0, 256, (1, n)).astype(np.uint8), False,
                           "MetropolisNonErgodic", 0)[:2]


def path(n):
    rng, h, u, v, J = problem(9)
    none = np.zeros(0, np.intc)
    return path_annealing(1, h, u, v, J, 1, [1.0], [0.5], 1.0, 0.0, 1, 1, 3,
                          workloads.random_states(rng, 1, 9), 1, 1, np.zeros((1, 9), np.intc), none,
                          none, 0, break_capacity=n)[:2]


def problem(n):
    rng = np.random.default_rng(n)
    u = np.arange(n - 1, dtype=np.int32)
    return rng, rng.normal(0, 0.3, n), u, u + 1, rng.normal(0, 1, n - 1)


@pytest.mark.parametrize("call,large,small", [(anneal, 4000, 200), (descent, 5000, 9),
                                              (rotor, 6000, 9), (path, 2000, 32)])
def test_two_sizes_at_once(call, large, small):
    want = {n: call(n) for n in (large, small)}
    wrong = []

    def work(n):
        try:
            for _ in range(60):
                for got, exp in zip(call(n), want[n]):
                    np.testing.assert_array_equal(got, exp)
        except Exception as x:  # noqa: BLE001 -- reported below
            wrong.append(x)

    threads = [threading.Thread(target=work, args=(n,)) for n in (large, small, small)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong
