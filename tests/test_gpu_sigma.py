"""The FP32 bound of a node's spectral radius (csrc/sigma.cuh): a node whose
FP64 value is the largest met so far must always be evaluated, whatever its
state -- low and hypersonic Mach numbers (pressure a millionth of the energy),
stretched cells, left-handed grids, areas whose squares leave FP32 -- and on
ordinary states the bound is tight enough to skip."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CSRC = Path(__file__).resolve().parents[1] / "cbns3d_cuda_b200" / "csrc"
SOURCE = r"""
#include "sigma.cuh"
using namespace cbns;
__global__ void k(const double* q, const double* A, const double* iJ, double* s, float* b, int* hit, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double Q[5], M[9];
  float qf[5], mf[9], small;
  for (int m = 0; m < 5; ++m) qf[m] = (float)(Q[m] = q[5 * i + m]);
  for (int m = 0; m < 9; ++m) mf[m] = (float)(M[m] = A[9 * i + m]);
  s[i] = sigma_exact(Q, M, iJ[i], 1.4, 0.4);
  b[i] = sigma_bound(qf, mf, (float)iJ[i], 1.4f, 0.4f, small);
  const bool one = sigma_reaches(b[i], small, __double2float_rd(s[i]));
  F2 q2[5], m2[9], sm2;
  for (int m = 0; m < 5; ++m) q2[m] = mk(qf[m], qf[m]);
  for (int m = 0; m < 9; ++m) m2[m] = mk(mf[m], mf[m]);
  const F2 b2 = sigma_bound(q2, m2, mk((float)iJ[i], (float)iJ[i]), 1.4f, 0.4f, sm2);
  float x, y, u, v;
  halves(b2, x, y);
  halves(sm2, u, v);
  hit[i] = one && sigma_reaches(x, u, __double2float_rd(s[i])) && sigma_reaches(y, v, __double2float_rd(s[i]));
}
template <typename T> static T* dev(size_t n) { T* d = nullptr; cudaMalloc(&d, n * sizeof(T)); return d; }
extern "C" int run(const double* q, const double* A, const double* iJ, double* s, float* b, int* hit, int n) {
  double *dq = dev<double>(5 * n), *dA = dev<double>(9 * n), *dJ = dev<double>(n), *ds = dev<double>(n);
  float* db = dev<float>(n); int* dh = dev<int>(n);
  cudaMemcpy(dq, q, 40 * (size_t)n, cudaMemcpyHostToDevice); cudaMemcpy(dA, A, 72 * (size_t)n, cudaMemcpyHostToDevice);
  cudaMemcpy(dJ, iJ, 8 * (size_t)n, cudaMemcpyHostToDevice);
  k<<<(n + 127) / 128, 128>>>(dq, dA, dJ, ds, db, dh, n);
  cudaMemcpy(s, ds, 8 * (size_t)n, cudaMemcpyDeviceToHost); cudaMemcpy(b, db, 4 * (size_t)n, cudaMemcpyDeviceToHost);
  const int e = cudaMemcpy(hit, dh, 4 * (size_t)n, cudaMemcpyDeviceToHost);
  cudaFree(dq); cudaFree(dA); cudaFree(dJ); cudaFree(ds); cudaFree(db); cudaFree(dh); return e;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("sigma")
    (d / "t.cu").write_text(SOURCE)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC", "-cudart", "static", "-I", str(CSRC), "-o", str(d / "t.so"), str(d / "t.cu")], check=True,
                   capture_output=True)
    return C.CDLL(str(d / "t.so"))


@pytest.mark.parametrize("kind", ["ordinary", "hypersonic", "still", "stretched", "tiny areas", "left-handed"])
def test_largest_node_is_always_evaluated(lib, kind):
    rng = np.random.default_rng(5)
    n = 200000
    rho = 10.0 ** rng.uniform(-1, 1, n)
    mach = {"hypersonic": 10.0 ** rng.uniform(1, 3, n), "still": np.zeros(n)}.get(kind, rng.uniform(0, 3, n))
    p = 10.0 ** rng.uniform(-1, 1, n)
    vel = rng.normal(size=(3, n))
    vel *= mach * np.sqrt(1.4 * p / rho) / np.sqrt((vel ** 2).sum(0))
    E = p / 0.4 + 0.5 * rho * (vel ** 2).sum(0)
    q = np.ascontiguousarray(np.stack([rho, *(rho * vel), E], -1))
    size = {"stretched": 10.0 ** rng.uniform(-6, 0, (n, 3, 1)), "tiny areas": 10.0 ** rng.uniform(-24, -14, (n, 3, 1))}
    A = np.ascontiguousarray((rng.normal(size=(n, 3, 3)) * size.get(kind, 1.0)).reshape(n, 9))
    iJ = 10.0 ** rng.uniform(-2, 4, n) * (-1.0 if kind == "left-handed" else 1.0)
    s, b, hit = np.empty(n), np.empty(n, np.float32), np.empty(n, np.int32)
    p_ = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    assert lib.run(p_(q), p_(A), p_(np.ascontiguousarray(iJ)), p_(s), p_(b), p_(hit), n) == 0
    assert np.isfinite(s).all() and (s > 0).all()
    assert hit.all()
    if kind == "ordinary":  # margins of 2e-5 and of 1e-6 E/p and 1e-6 |u|/c, a few at most here
        assert (b <= s * (1 + 1e-4)).all()
