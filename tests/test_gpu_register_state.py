"""Annealing with the state in registers, at the sizes where its variants
change (32, 64, 128, 256 variables), against the oracle: both orders and rules,
sparse and dense problems, spins other than +-1, betas that decide every
attempt alike, couplings of zero, one continued stream, several problems in a
launch."""
import numpy as np
import pytest

import oracle
from b200sa import sample_batch, simulated_annealing
from b200sa.workloads import Instance
from conftest import bits

pytestmark = pytest.mark.gpu

ORDERS = [(False, "Metropolis"), (False, "Gibbs"), (True, "Metropolis"), (True, "Gibbs")]


def problem(n, p, seed):
    rng = np.random.default_rng(seed)
    u, v = np.triu_indices(n, 1)
    keep = rng.random(len(u)) < p
    u, v = u[keep].astype(np.int32), v[keep].astype(np.int32)
    J = rng.normal(0, 1, len(u))
    J[rng.random(len(u)) < 0.1] = 0.0
    return rng, rng.normal(0, 0.4, n), u, v, J


def check(n, p, R, betas, order, rule, spins="pm1", shared=False, spb=1):
    rng, h, u, v, J = problem(n, p, n + int(100 * p))
    s0 = (rng.integers(-128, 128, (R, n)) if spins == "any"
          else 2 * rng.integers(0, 2, (R, n)) - 1).astype(np.int8)
    seeds = np.array([7]) if shared else 7 + np.arange(R)
    ws, we = oracle.run(h, u, v, J, s0, spb, betas, seeds.astype(np.uint64), order, rule == "Gibbs")
    st = {}
    s, e = simulated_annealing(R, h, u, v, J, spb, betas, 7, s0.copy(), order, rule,
                               rng_stream="shared" if shared else "per_read", stats=st)
    np.testing.assert_array_equal(s, ws)
    np.testing.assert_array_equal(bits(e), bits(we))
    assert st["near_ties"] == 0


@pytest.mark.parametrize("order,rule", ORDERS)
@pytest.mark.parametrize("n", [1, 2, 7, 31, 32, 33, 63, 64, 65, 96, 128, 129, 255, 256, 257,
                               320, 321])
@pytest.mark.parametrize("p", [0.08, 0.7])
def test_sizes(n, p, order, rule):
    check(n, p, 9, np.geomspace(0.02, 8.0, 12), order, rule, spb=2)


@pytest.mark.parametrize("order,rule", ORDERS)
@pytest.mark.parametrize("n", [20, 70, 200])
def test_any_spins(n, order, rule):
    check(n, 0.6, 5, np.geomspace(1e-4, 0.1, 8), order, rule, spins="any")


@pytest.mark.parametrize("order,rule", ORDERS)
def test_extreme_betas_and_continued_stream(order, rule):
    check(40, 0.5, 4, np.array([0.0, 1e-300, 1e3, 1e300]), order, rule, spb=3)
    check(90, 0.5, 6, np.geomspace(0.05, 5.0, 10), order, rule, shared=True)


def test_problems_of_one_launch():
    probs, want = [], []
    for k, (n, p, order, rule) in enumerate([(5, 1, 0, "Gibbs"), (30, 0.1, 0, "Gibbs"), (32, 1, 0, "Gibbs"),
                                             (120, 0.5, 0, "Gibbs"), (64, 0.2, 1, "Metropolis"),
                                             (250, 0.4, 1, "Metropolis"), (130, 0.9, 1, "Metropolis")]):
        rng, h, u, v, J = problem(n, p, 50 + k)
        R = 3 + k
        s0 = (2 * rng.integers(0, 2, (R, n)) - 1).astype(np.int8)
        betas, seeds = np.geomspace(0.1, 4.0, 9 + k), (11 * k + np.arange(R)).astype(np.uint64)
        want.append(oracle.run(h, u, v, J, s0, 1, betas, seeds, bool(order), rule == "Gibbs"))
        probs.append(Instance(h, u, v, J, s0.copy(), betas, 1, seeds, bool(order), rule))
    for mode in ("persistent", "plain"):
        got = [Instance(p.h, p.u, p.v, p.J, p.states.copy(), p.betas, 1, p.seeds, p.randomize_order,
                        p.proposal) for p in probs]
        en = sample_batch(got, mode=mode)
        for p, e, (ws, we) in zip(got, en, want):
            np.testing.assert_array_equal(p.states, ws)
            np.testing.assert_array_equal(bits(e), bits(we))
