"""Host-side packing, compiled for the CPU alone: what is packed for whom."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

WRAPPER = r"""
#include "pack.cpp"
extern "C" int64_t matrix_entries(int n, const double *h, int64_t m, const int32_t *u, const int32_t *v,
                                  const double *J, int reads, int betas) {
    b200sa_problem p{};
    p.num_vars = n;
    p.h = h;
    p.num_couplers = m;
    p.coupler_starts = u;
    p.coupler_ends = v;
    p.coupler_weights = J;
    p.num_reads = reads;
    p.sweeps_per_beta = 1;
    p.num_betas = betas;
    p.varorder = B200SA_SEQUENTIAL;
    b200sa::PackedAdjacency out;
    b200sa::pack_adjacency(p, out);
    return out.dense ? (int64_t)out.dense_w.size() : -(int64_t)out.dense_w.size();
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("pack")
    src, so = d / "wrap.cpp", d / "libpack.so"
    src.write_text(WRAPPER)
    inc = [os.path.join(ROOT, "include"), os.path.join(ROOT, "dwave-samplers_b200", "csrc"),
           "/usr/local/cuda/include"]
    subprocess.check_call(["g++", "-std=c++17", "-w", "-shared", "-fPIC", *(f"-I{i}" for i in inc), str(src),
                           "-o", str(so)])
    L = ctypes.CDLL(str(so))
    L.matrix_entries.restype = ctypes.c_int64
    return L


@pytest.mark.parametrize("n", [1, 2, 64, 65, 320])
def test_the_matrix_is_packed_for_annealing_alone(lib, n):
    """Steepest descent and the quantum samplers pass reads or none, and no schedule."""
    u, v = (x.astype(np.int32) for x in np.triu_indices(n, 1))
    h, J = np.zeros(n), np.ones(u.shape[0])

    def entries(reads, betas):
        return lib.matrix_entries(n, ctypes.c_void_p(h.ctypes.data), ctypes.c_int64(u.shape[0]),
                                  *(ctypes.c_void_p(a.ctypes.data) for a in (u, v, J)), reads, betas)

    assert entries(4, 3) > n * n
    assert entries(4, 0) == 0
    assert entries(0, 0) == 0
