"""The kernels' reciprocal (rcp_nr, csrc/cfk_common.cuh) against CUDA's own
division, over every binade whose reciprocal is a normal number.

Bar: 2 ulp of the correctly rounded quotient, the function's stated bound
(its last FMA rounds once, the truncated series leaves 2^-60)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROBE = """
#include "cfk_common.cuh"
__global__ void probe(const double *x, double *fast, double *quot, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  fast[i] = cfk::rcp_nr(x[i]);
  quot[i] = 1.0 / x[i];
}
extern "C" int run_probe(const double *x, double *fast, double *quot, int n) {
  probe<<<(n + 255) / 256, 256>>>(x, fast, quot, n);
  return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    import torch

    d = tmp_path_factory.mktemp("rcp")
    src, so = d / "rcp.cu", d / "rcp.so"
    src.write_text(PROBE)
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                    "-shared", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
                    "-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "corefl-cpc_b200", "csrc"),
                    str(src), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))

    def run(x):
        x = np.ascontiguousarray(x, dtype=np.float64)
        d = [torch.from_numpy(x).to("cuda:0"), torch.empty(x.size, dtype=torch.float64, device="cuda:0"),
             torch.empty(x.size, dtype=torch.float64, device="cuda:0")]
        torch.cuda.synchronize()
        assert lib.run_probe(*(ctypes.c_void_p(t.data_ptr()) for t in d), ctypes.c_int(x.size)) == 0
        return d[1].cpu().numpy(), d[2].cpu().numpy()

    return run


def _ulps(a, b):
    assert np.all(np.isfinite(a)) and np.all(np.sign(a) == np.sign(b))
    return np.abs(np.abs(a).view(np.int64) - np.abs(b).view(np.int64)).max()


def test_two_ulp_in_every_binade(probe):
    rng = np.random.default_rng(1)
    e = np.arange(-1022, 1022)  # [2^e, 2^(e+1)): reciprocals down to 2^-1022
    m = 1.0 + rng.integers(0, 2**52, size=(e.size, 256)) * 2.0**-52
    x = np.ldexp(m, e[:, None]).ravel()
    p = np.ldexp(1.0, e)
    x = np.concatenate([x, p, np.nextafter(p, np.inf), np.nextafter(p[1:], 0)])
    for s in (1.0, -1.0):
        fast, quot = probe(s * x)
        assert _ulps(fast, quot) <= 2


def test_edges_of_the_domain(probe):
    fast, quot = probe([0.0, -0.0, np.inf, -np.inf, np.nan])
    assert np.all(np.isnan(fast))  # a division gives inf or 0: the callers exclude these
    fast, quot = probe([2.0**-1022, -(2.0**-1022), 2.0**1021, 2.0**1022])
    assert _ulps(fast, quot) <= 2
