"""Device functions that stand in for CUDA's: the quotient by 2 pi of the table look-up (``over_twopi``)
against CUDA's division, bit for bit, and the lattice sums' exponential (``exp_neg``) against
extended precision.  They are compiled from the library's headers into a probe of their own."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROBE = r"""
#include "pss_lattice.cuh"
__global__ void k_probe(int n, const double *a, double *q, double *d, double *e) {
  __shared__ double tab[256];
  for (int t = threadIdx.x; t < 256; t += blockDim.x) tab[t] = exp2((double)t / 256.0);
  __syncthreads();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  q[i] = over_twopi(a[i]);
  d[i] = a[i] / PSS_TWOPI;
  e[i] = exp_neg(fabs(a[i]), tab);
}
extern "C" int probe(int n, const double *a, double *out) {
  double *da = nullptr, *dout = nullptr;
  if (cudaMalloc(&da, n * sizeof(double)) || cudaMalloc(&dout, 3 * (size_t)n * sizeof(double))) return 1;
  cudaMemcpy(da, a, n * sizeof(double), cudaMemcpyHostToDevice);
  k_probe<<<(n + 255) / 256, 256>>>(n, da, dout, dout + n, dout + 2 * (size_t)n);
  const int rc = (int)cudaMemcpy(out, dout, 3 * (size_t)n * sizeof(double), cudaMemcpyDeviceToHost);
  cudaFree(da);
  cudaFree(dout);
  return rc;
}
"""


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    d = tmp_path_factory.mktemp("probe")
    (d / "probe.cu").write_text(PROBE)
    subprocess.run([shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3",
                    "-std=c++17", "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-shared",
                    "-I", os.path.join(ROOT, "pssfss.jl_b200", "csrc"), "-I", os.path.join(ROOT, "include"),
                    "-o", str(d / "probe.so"), str(d / "probe.cu")], check=True)
    lib = ctypes.CDLL(str(d / "probe.so"))

    def run(a):
        a = np.ascontiguousarray(a, np.float64)
        out = np.zeros((3, len(a)))
        assert lib.probe(len(a), a.ctypes.data_as(ctypes.c_void_p), out.ctypes.data_as(ctypes.c_void_p)) == 0
        return out
    return run


def test_quotient_by_two_pi_is_correctly_rounded(probe):
    rng = np.random.default_rng(0)
    sign = lambda n: rng.choice([-1.0, 1.0], n)
    k = rng.integers(1, 4000, 200000) / rng.choice([1, 3, 7, 64, 400], 200000)
    near = k * 6.283185307179586  # quotients beside short fractions, where a last bit decides
    for _ in range(3):
        near = np.concatenate([near, np.nextafter(near[:200000], np.inf), np.nextafter(near[:200000], -np.inf)])
    a = np.concatenate([[0.0], sign(1000000) * rng.uniform(0, 30, 1000000),
                        sign(400000) * 10.0 ** rng.uniform(-250, 250, 400000), near * sign(len(near))])
    q, d, _ = probe(a)
    assert np.array_equal(q, d) and np.array_equal(d, a / 6.283185307179586)


def test_exponential_of_the_lattice_sums(probe):
    """Four units in the last place: two of CUDA's exp2 in the table, one of the polynomial, half of
    the product, and the argument's reduction, which is exact to 1e-20."""
    rng = np.random.default_rng(1)
    a = np.concatenate([[0.0], rng.uniform(0, 708, 400000), 10.0 ** rng.uniform(-20, 2.8, 400000),
                        np.arange(1, 200000) * (np.log(2) / 256)])  # and the ends of the reduction's steps
    a = a[a < 708.0]
    e = probe(a)[2]
    ref = np.exp(-a.astype(np.longdouble))
    assert float(np.max(np.abs(e - ref) / ref)) <= 4 * 2.0 ** -52
    assert np.all(probe(np.array([708.0, 800.0, 1e300]))[2] == 0.0)
