"""Windows whose flips share neighbours: hubs shared by a few and by all
variables, pairs and chains of variables with a common neighbour, equal and
unequal lists, state on chip and in global slots.  Every result equals the
oracle's."""
import numpy as np
import pytest

import oracle
from b200sa import simulated_annealing
from b200sa.sqa import simulated_annealing as rotor
from conftest import bits

pytestmark = pytest.mark.gpu


def graph(kind, n):
    rng = np.random.default_rng(n)
    if kind == "hub":  # every variable next to the last one
        u = np.arange(n - 1)
        v = np.full(n - 1, n - 1)
    elif kind == "hubs":  # groups of three variables share a distant one
        u = np.arange(n - n // 4)
        v = n - n // 4 + u // 3 % (n // 4)
    elif kind == "pairs":  # v and v + 2 share v + n / 2, which is next to v + 4 too
        h = n // 2
        i = np.arange(h)
        u = np.concatenate([i, i, i])
        v = h + np.concatenate([i, (i + 2) % h, (i + 4) % h])
    else:  # few targets for many sources
        u = np.repeat(np.arange(n - 40), 3)
        v = n - 40 + rng.integers(0, 40, len(u))
        key = np.unique(u * n + v)
        u, v = key // n, key % n
    return u.astype(np.int32), v.astype(np.int32), rng.normal(0, 0.7, len(u)), rng.normal(0, 0.3, n)


@pytest.mark.parametrize("rule", ["Metropolis", "Gibbs"])
@pytest.mark.parametrize("kind", ["hub", "hubs", "pairs", "few"])
@pytest.mark.parametrize("n,R", [(140, 5), (600, 40), (1500, 300)])
def test_shared_neighbours(kind, n, R, rule):
    u, v, J, h = graph(kind, n)
    s0 = (2 * np.random.default_rng(2).integers(0, 2, (R, n)) - 1).astype(np.int8)
    betas = np.array([0.02, 0.2, 0.7, 2.0])
    ws, we = oracle.run(h, u, v, J, s0, 1, betas, (3 + np.arange(R)).astype(np.uint64), False,
                        rule == "Gibbs")
    s, e = simulated_annealing(R, h, u, v, J, 1, betas, 3, s0.copy(), False, rule)
    np.testing.assert_array_equal(s, ws)
    np.testing.assert_array_equal(bits(e), bits(we))


@pytest.mark.parametrize("kind", ["hub", "pairs", "few"])
def test_reflections_share_neighbours(kind):
    n, R = 600, 20
    u, v, J, h = graph(kind, n)
    s0 = np.random.default_rng(2).integers(0, 256, (R, n)).astype(np.uint8)
    hp, hd, tf = np.array([0.02, 0.3, 2.0]), np.array([1.0, 0.5, 0.1]), np.ones(n)
    ws, we, _ = oracle.rotormc(h, u, v, J, tf, s0, 1, hp, hd, 4 + np.arange(R), False,
                               "MetropolisNonErgodic", 0)
    s, e, _ = rotor(R, h, u, v, J, tf, 1, hp, hd, 4, s0.copy(), False, "MetropolisNonErgodic", 0)
    np.testing.assert_array_equal(s, ws)
    np.testing.assert_array_equal(bits(e), bits(we))
