"""Where the FP64 values are formed by correctly rounded divisions and roots:

* the primitives that the stage kernels of a viscous run leave behind, to the
  bit: velocities as products with the rounded 1/rho, T = (gamma M^2 p)/rho;
* the spectral radius in FP64 (csrc/sigma.cuh), to the bit, against the same
  chain of single roundings in exact rational arithmetic.
"""
import ctypes as C
import math
import shutil
import subprocess
from fractions import Fraction
from pathlib import Path

import numpy as np
import pytest

import cbns3d_cuda_b200 as cb
from cbns3d_cuda_b200 import CBNS_Q, Block, cases, make_params

pytestmark = pytest.mark.gpu

CSRC = Path(__file__).resolve().parents[1] / "cbns3d_cuda_b200" / "csrc"
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
SOURCE = r"""
#include "sigma.cuh"
__global__ void k(const double* q, const double* A, const double* iJ, double* s, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) s[i] = cbns::sigma_exact(q + 5 * i, A + 9 * i, iJ[i], 1.4, 0.3999999999999999);
}
extern "C" int run(const double* q, const double* A, const double* iJ, double* s, int n) {
  double* d;
  cudaMalloc(&d, 128 * (size_t)n);
  cudaMemcpy(d, q, 40 * (size_t)n, cudaMemcpyHostToDevice);
  cudaMemcpy(d + 5 * n, A, 72 * (size_t)n, cudaMemcpyHostToDevice);
  cudaMemcpy(d + 14 * n, iJ, 8 * (size_t)n, cudaMemcpyHostToDevice);
  k<<<(n + 127) / 128, 128>>>(d, d + 5 * n, d + 14 * n, d + 15 * n, n);
  const int e = cudaMemcpy(s, d + 15 * n, 8 * (size_t)n, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e;
}
"""


@pytest.mark.parametrize("precision", [cb.PREC_FP64, cb.PREC_SPLIT])
def test_primitives_of_a_viscous_run(precision):
    (c,), _ = cases.case_batch(1, seed=7, size_lo=(40, 30, 20), size_hi=(41, 31, 21), viscous=True)
    c.params["bc_mode"] = cb.BC_FARFIELD
    with Block(make_params(*c.shape, **c.params, precision=precision)) as b:
        b.calc_metrics(c.x, c.y, c.z)
        b.set_conservative(c.Q0)
        b.calc_primitive(CBNS_Q)
        b.set_bc_calc_primitive(CBNS_Q)
        b.calc_viscous_terms()
        b.set_time(0.0)
        assert b.run(3) == 3
        inner = (slice(3, -3),) * 3
        shape = tuple(n + 4 for n in c.shape[::-1])
        q = b.get_conservative(CBNS_Q).reshape(shape + (5,))[inner]
        rho, u, v, w, p, T = (f.reshape(shape)[inner] for f in b.get_primitive())
        gM2 = b.p.gamma * (b.p.Mach * b.p.Mach)
    assert np.array_equal(rho, q[..., 0])
    for m, f in ((1, u), (2, v), (3, w)):
        assert np.array_equal(f, q[..., m] * (1.0 / rho))
    assert np.array_equal(T, gM2 * p / rho)


def _fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def _sigma(q, A, iJ, gamma, gam1):
    r, E = q[0], q[4]
    u, v, w = (q[m] * (1.0 / r) for m in (1, 2, 3))
    p = gam1 * _fma(-(0.5 * r), _fma(w, w, _fma(v, v, u * u)), E)
    c = math.sqrt(gamma * p / r)
    s = 0.0
    for d in range(3):
        x, y, z = (A[3 * d + m] * iJ for m in range(3))
        un = _fma(w, z, _fma(v, y, u * x))
        s += abs(un) + c * math.sqrt(_fma(z, z, _fma(y, y, x * x)))
    return s


def test_spectral_radius(tmp_path):
    if not Path(NVCC).exists():
        pytest.skip("compiles csrc/sigma.cuh with nvcc, which is not here")
    (tmp_path / "t.cu").write_text(SOURCE)
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC", "-cudart", "static", "-I", str(CSRC), "-o", str(tmp_path / "t.so"), str(tmp_path / "t.cu")],
                   check=True, capture_output=True)
    lib = C.CDLL(str(tmp_path / "t.so"))
    rng = np.random.default_rng(9)
    n = 3000
    rho, p = 10.0 ** rng.uniform(-1, 1, n), 10.0 ** rng.uniform(-1, 1, n)
    vel = rng.normal(size=(3, n))
    q = np.ascontiguousarray(np.stack([rho, *(rho * vel), p / 0.4 + 0.5 * rho * (vel ** 2).sum(0)], -1))
    A, iJ, s = rng.normal(size=(n, 9)), 10.0 ** rng.uniform(-2, 4, n) * rng.choice([-1.0, 1.0], n), np.empty(n)
    ptr = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    assert lib.run(ptr(q), ptr(A), ptr(iJ), ptr(s), n) == 0
    want = [_sigma(*a, 1.4, 0.3999999999999999) for a in zip(q.tolist(), A.tolist(), iJ.tolist())]
    assert np.array_equal(s, want)
