"""The face flux's own arithmetic on the GPU, from a small library compiled
against csrc/face_flux.cuh:

* FP64 reciprocal, reciprocal square root and square root against CUDA's
  1.0/x, rsqrt and sqrt, in units in the last place, over the exponent range a
  state meets and at special values;
* the FP32 face flux against the FP64 one on the same FP32 stencils: both
  branches of the tangent, smooth and jumping states, and jumps up to the
  largest the FP32 weights hold.
"""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CSRC = Path(__file__).resolve().parents[1] / "cbns3d_cuda_b200" / "csrc"
SOURCE = r"""
#include "face_flux.cuh"
using namespace cbns;
__global__ void k_math(const double* x, double* own, double* ref, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  own[i] = rcp_(x[i]); own[n + i] = rsqrt_(x[i]); own[2 * n + i] = sqrt_(x[i]);
  ref[i] = 1.0 / x[i]; ref[n + i] = rsqrt(x[i]); ref[2 * n + i] = sqrt(x[i]);
}
template <typename R>
__global__ void k_flux(const float* q, const float* nv, double* out, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  auto ld = [&](int p, int m) -> R { return (R)q[(i * 6 + p) * 5 + m]; };
  const FluxConsts<R> c{R(1.4), R(0.4), R(2.5)};
  R f[5];
  face_flux<R>(ld, (R)nv[3 * i], (R)nv[3 * i + 1], (R)nv[3 * i + 2], c, f);
  for (int m = 0; m < 5; ++m) out[i * 5 + m] = (double)f[m];
}
template <typename T> static T* up(const T* h, size_t n) {
  T* d = nullptr; cudaMalloc(&d, n * sizeof(T)); cudaMemcpy(d, h, n * sizeof(T), cudaMemcpyHostToDevice); return d;
}
extern "C" int run_math(const double* x, double* own, double* ref, int n) {
  double *dx = up(x, n), *a, *b; cudaMalloc(&a, 24 * (size_t)n); cudaMalloc(&b, 24 * (size_t)n);
  k_math<<<(n + 255) / 256, 256>>>(dx, a, b, n);
  cudaMemcpy(own, a, 24 * (size_t)n, cudaMemcpyDeviceToHost);
  const int e = cudaMemcpy(ref, b, 24 * (size_t)n, cudaMemcpyDeviceToHost);
  cudaFree(dx); cudaFree(a); cudaFree(b); return e;
}
extern "C" int run_flux(const float* q, const float* nv, double* f32, double* f64, int n) {
  float *dq = up(q, 30 * (size_t)n), *dn = up(nv, 3 * (size_t)n); double* o; cudaMalloc(&o, 40 * (size_t)n);
  k_flux<float><<<(n + 127) / 128, 128>>>(dq, dn, o, n);
  cudaMemcpy(f32, o, 40 * (size_t)n, cudaMemcpyDeviceToHost);
  k_flux<double><<<(n + 127) / 128, 128>>>(dq, dn, o, n);
  const int e = cudaMemcpy(f64, o, 40 * (size_t)n, cudaMemcpyDeviceToHost);
  cudaFree(dq); cudaFree(dn); cudaFree(o); return e;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("flux_math")
    (d / "t.cu").write_text(SOURCE)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC", "-cudart", "static", "-I", str(CSRC), "-o", str(d / "t.so"), str(d / "t.cu")], check=True,
                   capture_output=True)
    return C.CDLL(str(d / "t.so"))


def _p(a):
    return a.ctypes.data_as(C.c_void_p)


def test_fp64_reciprocal_and_roots(lib):
    rng = np.random.default_rng(1)
    n = 1 << 20
    # 32 orders of magnitude, and the neighbourhood of powers of two and of 1
    x = np.concatenate([10.0 ** rng.uniform(-16, 16, n - 4096), 2.0 ** rng.integers(-40, 40, 2048) * (1 + 2.0 ** -52 *
                       rng.integers(-4, 5, 2048)), 1 + 2.0 ** -52 * rng.integers(-1000, 1000, 2048)])
    own, ref = np.empty((3, n)), np.empty((3, n))
    assert lib.run_math(_p(x), _p(own), _p(ref), n) == 0
    ulp = np.abs(own - ref) / np.spacing(np.abs(ref))
    # the iteration leaves e^3 ~ 2^-58 and the rounding of its last step: 1 ulp;
    # sqrt = x rsqrt(x) adds a rounding; CUDA's own rsqrt is within 1 ulp
    assert ulp[0].max() <= 1 and ulp[1].max() <= 2 and ulp[2].max() <= 2
    s = np.array([-1.0, np.nan, 0.0, -4.0])
    own, ref = np.empty((3, 4)), np.empty((3, 4))
    assert lib.run_math(_p(s), _p(own), _p(ref), 4) == 0
    assert own[0, 0] == -1.0 and own[2, 2] == 0.0
    assert np.isnan(own[0, 1]) and np.isnan(own[1:, [0, 1, 3]]).all()


@pytest.mark.parametrize("kind", ["smooth", "jump", "axis", "huge"])
def test_fp32_flux_against_fp64(lib, kind):
    rng = np.random.default_rng(2)
    n = 20000
    if kind == "smooth":  # a wave of relative amplitude 1e-3 .. 0.1 along the stencil
        a = 10.0 ** rng.uniform(-3, -1, (n, 1))
        w = a * np.sin(rng.uniform(0, 6, (n, 1)) + 0.4 * np.arange(6))
    else:
        w = 0.4 * np.where(np.arange(6) < rng.integers(0, 7, (n, 1)), 1.0, -1.0)
    scale = 1.0e5 if kind == "huge" else 1.0
    rho, p = scale * (1 + w), scale * (0.7 + 0.6 * w)
    u, v, z = (rng.uniform(-1.5, 1.5, (n, 1)) + w for _ in range(3))
    E = p / 0.4 + 0.5 * rho * (u * u + v * v + z * z)
    q = np.ascontiguousarray(np.stack([rho, rho * u, rho * v, rho * z, E], -1).astype(np.float32))
    nv = rng.normal(size=(n, 3)).astype(np.float32)
    if kind == "axis":  # the tangent's other branch: the normal along x
        nv[:, 1:] = 0
    f32, f64 = np.empty((n, 5)), np.empty((n, 5))
    assert lib.run_flux(_p(q), _p(np.ascontiguousarray(nv)), _p(f32), _p(f64), n) == 0
    assert np.isfinite(f32).all() and np.isfinite(f64).all()
    # the flux's scale: energy times the largest signal speed times the area.
    # A reconstructed value is the centre state plus weights times differences;
    # 300 roundings of 6e-8 in the chain from the state to the weights
    qmax = np.abs(q).max(axis=(1, 2))
    c = np.sqrt(1.4 * p / rho).max(1) + np.sqrt(u * u + v * v + z * z).max(1)
    bound = 300 * 6.0e-8 * qmax * c * np.abs(nv).sum(1)
    assert (np.abs(f32 - f64).max(1) <= bound).all()
