"""Device memory of the buffer pool: a buffer takes what it needs, and what is
kept between calls stays below the pool's limit."""
import numpy as np
import pytest
import torch

import oracle
from b200sa import Plan, workloads
from b200sa.greedy import steepest_gradient_descent
from conftest import bits

pytestmark = pytest.mark.gpu

MB = 1 << 20


def problem(m, n=20000, seed=3):
    """40 bytes of adjacency and coupler records for each of m couplers."""
    rng = np.random.default_rng(seed)
    u = rng.integers(0, n // 2, m).astype(np.int32)
    v = rng.integers(n // 2, n, m).astype(np.int32)
    return workloads.Instance(rng.normal(0, 0.1, n), u, v, rng.normal(0, 1, m),
                              workloads.random_states(rng, 1, n), np.array([1.0]), 1,
                              np.arange(1, dtype=np.uint64) + 5)


def used():
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return (total - free) / MB


def test_a_buffer_takes_what_it_needs():
    with Plan([problem(1000)]):  # the context, the library's kernels
        pass
    before = used()
    m = 900_000  # 36 MB: above half of the largest block that is kept
    with Plan([problem(m)]):
        assert used() - before < 40 * m / MB + 10


def test_what_is_kept_stays_below_the_limit():
    base = used()
    for k in range(6):  # 50 to 60 MB each, 330 MB together
        m = int((50 + 2 * k) * MB / 40)
        with Plan([problem(m)]):
            pass
        assert used() - base < 256 + 20
    # Blocks of other sizes and contents serve the next call.
    rng = np.random.default_rng(1)
    h, s = rng.normal(0, 1, 30), workloads.random_states(rng, 5, 30)
    u = np.arange(29, dtype=np.int32)
    J = rng.normal(0, 1, 29)
    got, e, _ = steepest_gradient_descent(5, h, u, u + 1, J, s.copy())
    want, we, _ = oracle.descent(h, u, u + 1, J, s)
    np.testing.assert_array_equal(got, want)
    np.testing.assert_array_equal(bits(e), bits(we))
