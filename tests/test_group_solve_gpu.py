"""The lane-group kernels' 9 x 9 solve (group_solve, csrc/chem_fast.cuh) on its
own, ten systems a warp, against elimination in 80-bit arithmetic.

Bar: Gauss-Jordan with partial pivoting keeps the multipliers below 1, so the
elements grow by less than 2^8 (in fact by single digits), and the forward
error stays within the condition number times a few n eps: 200 cond 2^-53."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROBE = """
#include "chem_fast.cuh"
using namespace cfk;
__global__ void probe(const Mech *m, const double *A, const double *b, double *out) {
  const Lane<9, 3> me(*m, threadIdx.x);
  const int grp = me.base / 3;
  double a[3][9], x[9], y[3];
  for (int k = 0; k < 3; ++k)
    for (int r = 0; r < 9; ++r) a[k][r] = A[(grp * 9 + r) * 9 + k * 3 + me.j];
  for (int r = 0; r < 9; ++r) x[r] = b[grp * 9 + r];
  group_solve<9, 3>(a, x, me, y);
  if (me.own)
    for (int k = 0; k < 3; ++k) out[grp * 9 + k * 3 + me.j] = y[k];
}
extern "C" int run_probe(const double *A, const double *b, double *out) {
  void *m = nullptr;
  if (cudaMalloc(&m, sizeof(Mech)) != cudaSuccess || cudaMemset(m, 0, sizeof(Mech)) != cudaSuccess) return -1;
  probe<<<1, 32>>>(static_cast<const Mech *>(m), A, b, out);
  const int e = (int)cudaDeviceSynchronize();
  cudaFree(m);
  return e;
}
"""


@pytest.fixture(scope="module")
def solve(tmp_path_factory):
    import torch

    d = tmp_path_factory.mktemp("solve")
    src, so = d / "solve.cu", d / "solve.so"
    src.write_text(PROBE)
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                    "-shared", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
                    "-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "corefl-cpc_b200", "csrc"),
                    str(src), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))

    def run(A, b):
        assert A.shape == (10, 9, 9) and b.shape == (10, 9)
        d = [torch.from_numpy(np.ascontiguousarray(v)).to("cuda:0") for v in (A, b, np.zeros((10, 9)))]
        torch.cuda.synchronize()
        assert lib.run_probe(*(ctypes.c_void_p(t.data_ptr()) for t in d)) == 0
        return d[2].cpu().numpy()

    return run


def _exact(A, b):
    A, x = A.astype(np.longdouble), b.astype(np.longdouble)
    for i in range(9):
        p = i + int(np.argmax(np.abs(A[i:, i])))
        A[[i, p]], x[[i, p]] = A[[p, i]], x[[p, i]]
        for m in range(9):
            if m != i:
                f = A[m, i] / A[i, i]
                A[m] -= f * A[i]
                x[m] -= f * x[i]
    return x / np.diag(A)


def _check(solve, A, b):
    out = solve(A, b)
    for g in range(10):
        ref = _exact(A[g].copy(), b[g].copy())
        bar = 200 * np.linalg.cond(A[g], np.inf) * 2.0**-53
        assert np.abs(out[g] - ref).max() <= bar * np.abs(ref).max(), g


@pytest.mark.parametrize("t", [0.5, 1.0, 1.9, 3.9, 20.0])
def test_columns_below_the_diagonal(solve, t):
    """1 on the diagonal, -t below it, 1 in the last column: without row swaps
    the last column grows by (1 + t)^8, 3e5 at t = 3.9, and the solve loses
    that many digits; partial pivoting keeps it bounded for t > 1."""
    A = np.eye(9) - t * np.tril(np.ones((9, 9)), -1)
    A[:, -1] = 1.0
    rng = np.random.default_rng(3)
    _check(solve, np.stack([A] * 10), rng.normal(size=(10, 9)))


@pytest.mark.parametrize("pivots", ["all", "one", "none"])
def test_groups_of_a_warp_pivot_on_their_own(solve, pivots):
    """Random systems in the groups that pivot, diagonally dominant ones in
    the others, which the warp's swaps must leave alone."""
    rng = np.random.default_rng(7)
    for _ in range(20):
        A = rng.normal(size=(10, 9, 9))
        for g in range(10):
            if pivots == "none" or (pivots == "one" and g != 4):
                A[g] += 20 * np.eye(9)
            else:
                A[g] = A[g][rng.permutation(9)] * 10.0 ** rng.integers(-3, 4, size=(1, 9))
        _check(solve, A, rng.normal(size=(10, 9)))
