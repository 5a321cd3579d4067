"""A stream captured by one thread while another one calls the samplers: the
calls wait for their own work alone, so the capture goes on and both results
are right.  The calls are made twice, with buffers new and kept."""
import threading

import numpy as np
import pytest
import torch

from b200sa import sample_batch, simulated_annealing, workloads
from b200sa.greedy import steepest_gradient_descent
from b200sa.sqa import path_annealing
from b200sa.sqa import simulated_annealing as rotor_annealing

pytestmark = pytest.mark.gpu


def problem(n, reads):
    rng = np.random.default_rng(n)
    u = np.arange(n - 1, dtype=np.int32)
    return rng.normal(0, 0.3, n), u, u + 1, rng.normal(0, 1, n - 1), workloads.random_states(rng, reads, n)


def anneal(n=40):
    h, u, v, J, s = problem(n, 7)
    return simulated_annealing(7, h, u, v, J, 1, [0.5, 1.0, 2.0], 3, s)


def global_slots():
    return anneal(9000)


def batch():
    ps = []
    for n in (30, 700):
        h, u, v, J, s = problem(n, 5)
        ps.append(workloads.Instance(h, u, v, J, s, np.array([0.5, 1.0]), 1, np.arange(1, 6, dtype=np.uint64)))
    return [*sample_batch(ps), *(p.states for p in ps)]


def descent():
    h, u, v, J, s = problem(60, 7)
    return steepest_gradient_descent(7, h, u, v, J, s)


def rotor():
    h, u, v, J, s = problem(40, 7)
    return rotor_annealing(7, h, u, v, J, np.ones(40), 1, [0.5, 1.0], [0.5, 0.1], 3,
                           (s + 1).astype(np.uint8), False, "MetropolisTF", 0)[:2]


def path():
    h, u, v, J, s = problem(40, 7)
    none = np.zeros(0, np.intc)
    return path_annealing(7, h, u, v, J, 1, [0.5, 1.0], [2.0, 0.1], 1.0, 0.0, 1, 1, 3, s, 1, 1,
                          np.zeros((7, 40), np.intc), none, none, 0)[:2]


@pytest.mark.parametrize("call", [anneal, global_slots, batch, descent, rotor, path])
def test_calls_beside_a_capture(call):
    want = call()
    got = []

    def work():
        try:
            got.extend([call(), call()])
        except Exception as x:  # noqa: BLE001 -- reported below
            got.append(x)

    x = torch.zeros(8, device="cuda")
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
        x.add_(1.0)
        t = threading.Thread(target=work)
        t.start()
        t.join()
        x.add_(2.0)
    graph.replay()
    torch.cuda.synchronize()
    assert (x == 3.0).all()
    assert len(got) == 2, got
    for res in got:
        for a, b in zip(res, want):
            np.testing.assert_array_equal(a, b)
