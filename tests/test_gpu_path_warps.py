"""Path-integral annealing by a warp per sample: break lists and
interface lists shorter and longer than a warp, ties between them, self-loops
and repeated couplers, high degrees, sample counts that leave
a CTA partly empty.  Every result equals the oracle's."""
import ctypes

import numpy as np
import pytest

import oracle
from b200sa import _lib
from conftest import bits

pytestmark = pytest.mark.gpu


def run(n, m, R, hd, hp, spb=1, quantum=False, seed=5, shared=False):
    rng = np.random.default_rng(seed)
    u, v = (rng.integers(0, n, m).astype(np.int32) for _ in range(2))
    J, h = rng.normal(0, 1, m), rng.normal(0, 0.3, n)
    s0 = (2 * rng.integers(0, 2, (R, n)) - 1).astype(np.int8)
    hp, hd = np.asarray(hp, float), np.asarray(hd, float)
    nb = np.zeros((R, n), np.intc)
    lists = np.zeros(0, np.intc)
    if quantum:  # even counts, equal neighbours among them
        nb = (2 * rng.integers(0, 8, (R, n))).astype(np.intc)
        lists = np.concatenate([np.sort(rng.integers(0, 65536, k)) // 4096 * 4096 if k % 4 else
                                np.sort(rng.integers(0, 65536, k)) for k in nb.ravel()]).astype(np.intc)
    nb_in = nb.copy()
    st, en = s0.copy(), np.empty(R)
    seeds = (np.array([seed]) if shared else seed + np.arange(R)).astype(np.uint32)
    out = np.zeros(max(1, R * n * 256), np.intc)
    near, err = ctypes.c_int64(0), _lib.errbuf()
    cap = int(np.ceil(hd.max() + 10 * np.sqrt(hd.max()) + 32)) if len(hd) else 16
    rc = _lib.load().b200sa_path_anneal(
        n, h.ctypes.data, m, u.ctypes.data, v.ctypes.data, J.ctypes.data, R, st.ctypes.data,
        en.ctypes.data, spb, len(hd), hp.ctypes.data, hd.ctypes.data, 0.0, 1, 1,
        seeds.ctypes.data, len(seeds), 0 if quantum else 1, 0, nb.ctypes.data,
        lists.ctypes.data, len(lists), out.ctypes.data, len(out), None, 0, cap, 0,
        ctypes.byref(near), err, len(err))
    _lib.check(rc, err)
    assert near.value == 0
    return h, u, v, J, s0, hp, hd, nb_in, lists, st, en, nb, out


def check(n, m, R, hd, hp, quantum=False, shared=False, **kw):
    h, u, v, J, s0, hp, hd, nb_in, lists, st, en, nb, out = run(n, m, R, hd, hp, quantum=quantum,
                                                                shared=shared, **kw)
    spb, seed = kw.get("spb", 1), kw.get("seed", 5)
    offs = np.concatenate([[0], np.cumsum(nb_in.sum(axis=1))])
    rows = [(0, R)] if shared else [(r, r + 1) for r in range(R)]
    pos = 0
    for a, b in rows:
        extra = dict(num_breaks=nb_in[a:b], breaks_in=lists[offs[a]:offs[b]]) if quantum else {}
        ws, we, _, wnb, wl = oracle.pimc(h, u, v, J, s0[a:b], spb, hp, hd, seed if shared else seed + a,
                                         0.0, 1, 1, not quantum, False, max_out=256, **extra)
        np.testing.assert_array_equal(st[a:b], ws)
        np.testing.assert_array_equal(bits(en[a:b]), bits(we))
        np.testing.assert_array_equal(nb[a:b], wnb)
        flat = wl[np.arange(256) < wnb[:, :, None]]
        np.testing.assert_array_equal(out[pos:pos + len(flat)], flat)
        pos += len(flat)


@pytest.mark.parametrize("n,m,R", [(1, 0, 3), (2, 3, 5), (9, 40, 33), (64, 1500, 7), (40, 100, 130)])
@pytest.mark.parametrize("gamma", [0.0, 0.3, 6.0, 40.0])
def test_lists_around_a_warp(n, m, R, gamma):
    check(n, m, R, [gamma, gamma / 2, gamma / 7], [0.2, 1.0, 4.0], spb=2)


def test_many_samples():
    check(3, 4, 5000, [2.0, 0.5], [0.5, 2.0])


@pytest.mark.parametrize("seed", [1, 2])
def test_quantum_states_with_equal_breaks(seed):
    check(20, 60, 9, [5.0, 5.0, 1.0], [0.3, 1.0, 2.0], quantum=True, seed=seed)


def test_continued_stream():
    check(16, 40, 6, [4.0, 1.0], [0.5, 2.0], shared=True, spb=2)
