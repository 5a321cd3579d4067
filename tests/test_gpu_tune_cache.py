"""The tuning cache: what its keys tell apart, and entries that do not fit."""
import numpy as np
import pytest
import torch

from b200sa import Plan, workloads

pytestmark = pytest.mark.gpu


def problem(n, u, v, reads, seed):
    rng = np.random.default_rng(seed)
    return workloads.Instance(rng.normal(0, 0.1, n), u.astype(np.int32), v.astype(np.int32),
                              rng.normal(0, 1, u.shape[0]), workloads.random_states(rng, reads, n),
                              np.geomspace(0.1, 3.0, 6), 1, np.arange(reads, dtype=np.uint64) + 5)


def ring(n, reads=8):
    """Every list two entries long."""
    return problem(n, np.arange(n), (np.arange(n) + 1) % n, reads, 1)


def path(n, reads=8):
    """The same mean degree, rounded, with two shorter lists."""
    return problem(n, np.arange(n - 1), np.arange(1, n), reads, 2)


def run(plan, p):
    sin = torch.from_numpy(p.states.ravel()).cuda()
    out, en = torch.empty_like(sin), torch.empty(plan.total_reads, dtype=torch.float64, device="cuda")
    plan.run(sin, out, en)
    return out, en


def keys(cache):
    return [line.split()[0] for line in cache.read_text().splitlines()]


def test_equal_and_unequal_lists_have_entries_of_their_own(tmp_path):
    cache = tmp_path / "tune.txt"
    for p in (ring(300), path(300)):
        with Plan([p]) as plan:
            assert [e["from_cache"] for e in plan.autotune(str(cache))] == [0]
    assert len(set(keys(cache))) == 2


def test_entries_of_other_sources_are_not_taken(tmp_path):
    from build import digest
    cache = tmp_path / "tune.txt"
    with Plan([ring(300)]) as plan:
        plan.autotune(str(cache))
    text = cache.read_text()
    assert f";src={digest()};" in text
    cache.write_text(text.replace(digest(), "0" * 12))
    with Plan([ring(300)]) as plan:
        assert [e["from_cache"] for e in plan.autotune(str(cache))] == [0]


@pytest.mark.parametrize("staging,n", [(3, 20000), (1, 2000), (2, 15000)])
def test_an_entry_that_does_not_fit_is_measured_anew(tmp_path, staging, n):
    """16 regions do not fit a CTA in any of these."""
    cache = tmp_path / "tune.txt"
    p = ring(n)
    with Plan([p]) as plan:
        ref, en_ref = run(plan, p)
        plan.autotune(str(cache))
    cache.write_text("".join(f"{k} {staging} 16 0 0 1.0\n" for k in keys(cache)))
    with Plan([p]) as plan:
        rep = plan.autotune(str(cache))
        assert [e["from_cache"] for e in rep] == [0] and rep[0]["candidates"] > 0
        out, en = run(plan, p)
        assert torch.equal(out, ref) and torch.equal(en, en_ref)
    assert f" {staging} 16 0 0 1\n" not in cache.read_text()
