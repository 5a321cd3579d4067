"""Device buffers and streams reused between calls: calls of changing sizes
from several threads at once, plans closed while others run, and buffers of a
failed call."""
import threading

import numpy as np
import pytest

import oracle
from b200sa import Plan, sample_batch, simulated_annealing, workloads
from b200sa.greedy import steepest_gradient_descent
from conftest import bits

pytestmark = pytest.mark.gpu


def small(n, seed, reads):
    rng = np.random.default_rng(seed)
    u = np.arange(n - 1, dtype=np.int32)
    return workloads.Instance(rng.normal(0, 0.3, n), u, u + 1, rng.normal(0, 1, n - 1),
                              workloads.random_states(rng, reads, n), np.geomspace(0.2, 3.0, 7), 1,
                              np.arange(seed, seed + reads, dtype=np.uint64))


def test_threads_and_sizes():
    wrong = []

    def work(t):
        try:
            for k in range(6):
                p = small(20 + 97 * ((t + k) % 5), 100 * t + k, 3 + 40 * (k % 3))
                ws, we = oracle.run(p.h, p.u, p.v, p.J, p.states, 1, p.betas, p.seeds)
                if k % 2:
                    q = workloads.Instance(p.h, p.u, p.v, p.J, p.states.copy(), p.betas, 1, p.seeds)
                    e = sample_batch([q, small(70, t, 5)])[0]
                    s = q.states
                else:
                    s, e = simulated_annealing(p.num_reads, p.h, p.u, p.v, p.J, 1, p.betas, 0,
                                               p.states.copy(), seeds=p.seeds)
                np.testing.assert_array_equal(s, ws)
                np.testing.assert_array_equal(bits(e), bits(we))
        except Exception as x:  # noqa: BLE001 -- reported below
            wrong.append(x)

    threads = [threading.Thread(target=work, args=(t,)) for t in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong


def test_closing_plans_while_another_runs():
    import torch
    p = small(900, 5, 64)
    p.betas = np.geomspace(0.2, 3.0, 300)
    keep = Plan([p, small(60, 6, 9)])
    sin = torch.from_numpy(np.concatenate([p.states.ravel(), small(60, 6, 9).states.ravel()])).cuda()
    want = torch.empty_like(sin)
    en = torch.empty(keep.total_reads, dtype=torch.float64, device="cuda")
    keep.run(sin, want, en)
    for _ in range(4):
        out = torch.zeros_like(sin)
        keep.run(sin, out, en, stream=torch.cuda.current_stream(), sync=False)
        for k in range(3):  # their buffers and streams come back and go out again
            Plan([small(50 + k, k, 11)]).close()
            simulated_annealing(2, [0.1], [], [], [], 1, [1.0], 3, np.ones((2, 1), np.int8))
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    keep.close()


def test_buffers_of_a_failed_call_come_back():
    with pytest.raises(TimeoutError):  # a positive self-loop makes descent cycle
        steepest_gradient_descent(4, [0.0], [0], [0], [1.0], np.ones((4, 1), np.int8), max_steps=50)
    s, e, k = steepest_gradient_descent(4, [1.0], [], [], [], np.ones((4, 1), np.int8))
    assert (s == -1).all() and (e == -1.0).all() and (k == 1).all()
