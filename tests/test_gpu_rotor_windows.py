"""Rotor-model annealing at the edges of its windows: sizes around 7 and 32
variables, repeated couplers and self-loops, neighbours one apart, every state
location, the schedule's extremes.  Every result equals the oracle's bit for
bit."""
import numpy as np
import pytest

import oracle
from b200sa.sqa import simulated_annealing
from conftest import bits

pytestmark = pytest.mark.gpu


def problem(n, graph, seed):
    rng = np.random.default_rng(seed)
    if graph == "none":
        u = v = np.zeros(0, np.int32)
    elif graph == "chain":
        u = np.arange(max(n - 1, 0), dtype=np.int32)
        v = u + 1
    elif graph == "dense":
        u, v = (x.astype(np.int32) for x in np.triu_indices(n, 1))
    else:  # repeated couplers and self-loops among them
        u = rng.integers(0, n, 3 * n).astype(np.int32)
        v = rng.integers(0, n, 3 * n).astype(np.int32)
    return rng, u, v, rng.normal(0, 1, len(u)), rng.normal(0, 0.3, n), rng.uniform(0, 2, n)


def check(n, graph, proposal, order, R=5, spb=1, betas=6, hp=None, hd=None, shared=False):
    rng, u, v, J, h, tf = problem(n, graph, n + 7)
    hp = np.geomspace(0.1, 40.0, betas) if hp is None else np.asarray(hp, float)
    hd = np.geomspace(20.0, 0.01, len(hp)) if hd is None else np.asarray(hd, float)
    st0 = rng.integers(0, 256, (R, n)).astype(np.uint8)
    with np.errstate(all="ignore"):
        ws, we, wst = oracle.rotormc(h, u, v, J, tf, st0, spb, hp, hd,
                                     [91] if shared else 91 + np.arange(R), order, proposal, 2)
        s, e, st = simulated_annealing(R, h, u, v, J, tf, spb, hp, hd, 91, st0.copy(), order,
                                       proposal, 2, rng_stream="shared" if shared else "per_read")
    np.testing.assert_array_equal(s, ws)
    np.testing.assert_array_equal(bits(e), bits(we))
    if not shared:
        np.testing.assert_array_equal(st, wst)


@pytest.mark.parametrize("proposal", list(oracle.ROTOR_PROPOSALS))
@pytest.mark.parametrize("order", [False, True])
@pytest.mark.parametrize("n,graph", [(1, "none"), (1, "loops"), (6, "dense"), (7, "chain"),
                                     (8, "loops"), (31, "chain"), (32, "dense"), (33, "chain"),
                                     (65, "loops"), (100, "dense")])
def test_window_edges(n, graph, proposal, order):
    check(n, graph, proposal, order)


@pytest.mark.parametrize("proposal", list(oracle.ROTOR_PROPOSALS))
@pytest.mark.parametrize("order", [False, True])
@pytest.mark.parametrize("n,R", [(2500, 3600), (270000, 2)])
def test_state_locations(n, R, proposal, order):
    # Spins on chip beside global delta energies; everything in global slots
    # (and, in random order, the bitmap too).
    if n > 100000:
        check(n, "chain", proposal, order, R=R, betas=2)
    else:
        check(n, "loops", proposal, order, R=R, betas=1)


@pytest.mark.parametrize("proposal", list(oracle.ROTOR_PROPOSALS))
@pytest.mark.parametrize("order", [False, True])
def test_schedule_extremes_and_continued_stream(proposal, order):
    check(40, "loops", proposal, order, hp=[1e-300, 1.0, 1e300, 0.0, -1.0],
          hd=[1.0, 1e-9, 1.0, 0.5, 0.25])
    check(40, "loops", proposal, order, spb=3, shared=True)


@pytest.mark.parametrize("proposal", ["MetropolisUniform", "MetropolisTF"])
@pytest.mark.parametrize("order", [False, True])
def test_one_thread_per_sample(proposal, order):
    check(9, "loops", proposal, order, R=20001, betas=3)
