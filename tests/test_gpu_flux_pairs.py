"""The face flux of two faces in packed FP32 (csrc/face_flux.cuh, F2), the form
the split and hybrid kernels run, against the FP64 flux on the same FP32
stencils.  The two faces of a pair differ in state, size and normal: one may
take the tangent's other branch (a normal along x) beside one that does not.

* mixed: waves and jumps of ordinary states;
* ramp, jump: differences from node to node up to 5e8, where the squares of the
  smoothness indicators' products are far beyond the FP32 range.

The bound is per component: 300 roundings of 6e-8 in the chain from the state
to the weights, times the flux's scale, the largest energy E of the stencil
times the largest signal speed a times the area -- over c^2 for the mass, c for
the momentum (c the least speed of sound).
"""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CSRC = Path(__file__).resolve().parents[1] / "cbns3d_cuda_b200" / "csrc"
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
SOURCE = r"""
#include "face_flux.cuh"
using namespace cbns;
__global__ void k_pair(const float* q, const float* nv, double* out, int pairs) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= pairs) return;
  const float *q0 = q + 60 * (size_t)i, *q1 = q0 + 30, *n0 = nv + 6 * (size_t)i, *n1 = n0 + 3;
  auto ld = [&](int p, int m) -> F2 { return mk(q0[5 * p + m], q1[5 * p + m]); };
  const FluxConsts<float> c{1.4f, 0.4f, 2.5f};
  F2 f[5];
  face_flux<F2>(ld, mk(n0[0], n1[0]), mk(n0[1], n1[1]), mk(n0[2], n1[2]), c, f);
  for (int m = 0; m < 5; ++m) {
    float a, b;
    halves(f[m], a, b);
    out[10 * (size_t)i + m] = a;
    out[10 * (size_t)i + 5 + m] = b;
  }
}
template <typename R>
__global__ void k_one(const float* q, const float* nv, double* out, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  auto ld = [&](int p, int m) -> R { return (R)q[30 * (size_t)i + 5 * p + m]; };
  const FluxConsts<R> c{R(1.4), R(0.4), R(2.5)};
  R f[5];
  face_flux<R>(ld, (R)nv[3 * i], (R)nv[3 * i + 1], (R)nv[3 * i + 2], c, f);
  for (int m = 0; m < 5; ++m) out[5 * (size_t)i + m] = (double)f[m];
}
extern "C" int run(const float* q, const float* nv, double* out, int n) {  // out: pairs, FP32, FP64
  float *dq, *dn;
  double* o;
  cudaMalloc(&dq, 120 * (size_t)n);
  cudaMalloc(&dn, 12 * (size_t)n);
  cudaMalloc(&o, 120 * (size_t)n);
  cudaMemcpy(dq, q, 120 * (size_t)n, cudaMemcpyHostToDevice);
  cudaMemcpy(dn, nv, 12 * (size_t)n, cudaMemcpyHostToDevice);
  k_pair<<<(n / 2 + 127) / 128, 128>>>(dq, dn, o, n / 2);
  k_one<float><<<(n + 127) / 128, 128>>>(dq, dn, o + 5 * (size_t)n, n);
  k_one<double><<<(n + 127) / 128, 128>>>(dq, dn, o + 10 * (size_t)n, n);
  const int e = cudaMemcpy(out, o, 120 * (size_t)n, cudaMemcpyDeviceToHost);
  cudaFree(dq);
  cudaFree(dn);
  cudaFree(o);
  return e;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if not Path(NVCC).exists():
        pytest.skip("compiles csrc/face_flux.cuh with nvcc, which is not here")
    d = tmp_path_factory.mktemp("flux_pairs")
    (d / "t.cu").write_text(SOURCE)
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC", "-cudart", "static", "-I", str(CSRC), "-o", str(d / "t.so"), str(d / "t.cu")], check=True,
                   capture_output=True)
    return C.CDLL(str(d / "t.so"))


@pytest.mark.parametrize("kind", ["mixed", "ramp", "jump"])
def test_both_faces_of_a_pair(lib, kind):
    rng = np.random.default_rng(3)
    n = 40000
    step = np.where(np.arange(6) < rng.integers(0, 7, (n, 1)), 1.0, -1.0)
    wave = 10.0 ** rng.uniform(-3, -1, (n, 1)) * np.sin(rng.uniform(0, 6, (n, 1)) + 0.4 * np.arange(6))
    size = 10.0 ** rng.uniform(0, 8.7, (n, 1))
    shape = {"mixed": np.where(rng.random((n, 1)) < 0.5, 1 + 0.4 * step, 1 + wave), "jump": size * (1 + 0.4 * step),
             "ramp": 1 + size * np.where(rng.random((n, 1)) < 0.5, np.arange(6), 5 - np.arange(6))}[kind]
    rho, p = shape, 0.7 * shape
    if kind == "mixed":
        p = p * (1 + 0.2 * rng.uniform(-1, 1, (n, 1)) * (shape - 1))
    u, v, z = (rng.uniform(-1.5, 1.5, (n, 1)) + (0.1 * step if kind != "ramp" else 0.0) for _ in range(3))
    E = p / 0.4 + 0.5 * rho * (u * u + v * v + z * z)
    q = np.ascontiguousarray(np.stack([rho, rho * u, rho * v, rho * z, E], -1).astype(np.float32))
    nv = rng.normal(size=(n, 3)).astype(np.float32)
    nv[rng.random(n) < 0.3, 1:] = 0  # the tangent's other branch, beside either
    nv = np.ascontiguousarray(nv)
    out = np.empty((3, n, 5))
    assert lib.run(q.ctypes.data_as(C.c_void_p), nv.ctypes.data_as(C.c_void_p), out.ctypes.data_as(C.c_void_p), n) == 0
    assert np.isfinite(out).all()
    speed = np.sqrt(u * u + v * v + z * z)
    c = np.sqrt(1.4 * p / rho)
    scale = E.max(1) * (c.max(1) + speed.max(1)) * np.abs(nv).sum(1)
    least = c.min(1)
    bound = 300 * 6.0e-8 * np.stack([scale / least ** 2, *[scale / least] * 3, scale], -1)
    for fp32 in out[:2]:
        assert (np.abs(fp32 - out[2]) <= bound).all()
