"""Windows whose variables neighbour each other, solved together in a pass:
chains, lattices whose rows are shorter, equal and longer than a window, dense
problems above the register sizes; hot and cold, both rules, every state
location of such problems.  Every result equals the oracle's."""
import numpy as np
import pytest

import oracle
from b200sa import simulated_annealing, workloads
from conftest import bits

pytestmark = pytest.mark.gpu


def graph(kind, size):
    rng = np.random.default_rng(size)
    if kind == "chain":
        u = np.arange(size - 1, dtype=np.int32)
        return size, u, u + 1, rng.normal(0, 1, size - 1)
    if kind == "lattice":
        p = workloads.cubic_lattice(L=size, reads=1, sweeps=1, seed=size)
        return size ** 3, p.u, p.v, p.J * rng.uniform(0.5, 1.5, len(p.J))
    u, v = (x.astype(np.int32) for x in np.triu_indices(size, 1))
    if kind == "near":  # up to four of the next 40 variables
        keep = (v - u <= 40) & (rng.random(len(u)) < 0.1)
        u, v = u[keep], v[keep]
    return size, u, v, rng.normal(0, 0.3, len(u))


@pytest.mark.parametrize("rule", ["Metropolis", "Gibbs"])
@pytest.mark.parametrize("kind,size,R", [("chain", 129, 9), ("chain", 2001, 300), ("lattice", 6, 20),
                                         ("lattice", 11, 9), ("lattice", 21, 3), ("lattice", 22, 3),
                                         ("lattice", 32, 2),
                                         ("dense", 330, 5), ("near", 400, 20), ("near", 9000, 3)])
def test_resolved_windows(kind, size, R, rule):
    n, u, v, J = graph(kind, size)
    rng = np.random.default_rng(1)
    h = rng.normal(0, 0.2, n)
    s0 = (2 * rng.integers(0, 2, (R, n)) - 1).astype(np.int8)
    s0[-1] = -1
    if R > 2:
        s0[0, 0] = 3  # a read with another spin value beside the others
    betas = np.array([0.01, 0.1, 0.4, 1.0, 3.0, 30.0])
    seeds = (5 + np.arange(R)).astype(np.uint64)
    ws, we = oracle.run(h, u, v, J, s0, 1, betas, seeds, False, rule == "Gibbs")
    st = {}
    s, e = simulated_annealing(R, h, u, v, J, 1, betas, 5, s0.copy(), False, rule, stats=st)
    np.testing.assert_array_equal(s, ws)
    np.testing.assert_array_equal(bits(e), bits(we))
    assert st["near_ties"] == 0
