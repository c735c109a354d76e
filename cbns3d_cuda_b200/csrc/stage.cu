// stage.cu - one SSP-RK3 stage in one kernel: inviscid WENO5-char/LF fluxes in
// all three directions, their differences, the viscous divergence (formed
// ahead of it by visc_div_kernel, visc.cu), division by J and the Shu-Osher
// stage combination, for every interior node.
//
// Replaces, for one stage, the reference's
//   calc_numerical_flux  (src/calc_numerical_flux.cu:15-74; three face kernels
//                         writing Ep/Fp/Gp to HBM)
//   update_rk3 / rk3_kernel     (src/time_integration.cu:15-40,
//                                src/runge_kutta_kernel.cu:13-80)
// and, in stage 3 of an inviscid step, the per-node half of calc_dt
// (src/time_step_kernel.cu:13-96) for interior nodes.
//
// Tiling (2.5D).  A CTA of 256 threads owns a TI x TJ = 16 x 15 column of
// interior nodes and marches it through a chunk of k planes.  Per plane:
//   ring   : the conservative state of the column on the 6 planes k-2..k+3
//            (stencil of the k-faces), loaded one new plane per step;
//   plane  : plane k with a 3-node halo in i and j (stencils of i/j faces);
//   areas  : the node area vectors J*grad(xi) on the i-face nodes and
//            J*grad(eta) on the j-face nodes of plane k (face normals);
//   round A: the 17 x 15 i-faces of plane k  (thread f -> face f, f < 255)
//   round B: the 16 x 16 j-faces of plane k  (thread f -> face f)
//   round C: the k+1/2 face of each column   (thread t -> column t, t < 240);
//            the k-1/2 flux and the column's J*grad(zeta) are carried in
//            registers from the previous plane.
// Every thread computes 3 faces per plane; face fluxes never leave the SM and
// no global load sits inside a face evaluation.  This is the FP64 kernel; the
// FP32-flux precisions run stage32.cu.
// HBM traffic per node and stage: the stage input (40 B, halos from L2), area
// vectors and 1/J (80 B), the RK base (0-40 B) and the output (40 B).
#include <mutex>

#include "cbns_common.cuh"
#include "face_flux.cuh"
#include "sigma.cuh"
#include "stage.cuh"
#include "tma.cuh"

namespace cbns {

namespace {

constexpr int TI = STAGE_TI, TJ = STAGE_TJ, H = 3;
constexpr int PW = TI + 2 * H;  // 22
constexpr int PH = TJ + 2 * H;  // 21
constexpr int NC = TI * TJ;     // 240 columns
constexpr int NT = 256;         // threads
constexpr int NFI = (TI + 1) * TJ;  // 255 i-faces
constexpr int NFJ = TI * (TJ + 1);  // 256 j-faces
// the face rounds' thread mapping (face_a, face_b in stage_body): one j-face
// per thread; i-faces on 7 warps of two 16-face rows and one of a row and the
// 15 faces of the last column
static_assert(NFJ == NT && TI == 16 && TJ == 15, "face mapping of the face rounds");
static_assert(NFI == 7 * 32 + 16 + TJ, "face mapping of the face rounds");
constexpr int NSX = (TI + 2) * TJ;  // i-face nodes (i0-1 .. i0+16)
constexpr int NSY = TI * (TJ + 2);  // j-face nodes (j0-1 .. j0+15)
constexpr int NHI = 2 * H * TJ, NHJ = 2 * H * TI;  // halo nodes of a plane: i-halo, j-halo

// x / 3: the product with the rounded 1/3 corrected by its exact residual,
// three operations for the division's dozen (the residual x - 3q is exact, so
// the result is x/3 rounded once more).
__device__ __forceinline__ double third(double x) {
  const double q = ml(x, 1.0 / 3.0);
  return fm(fm(-3.0, q, x), 1.0 / 3.0, q);
}

__device__ __forceinline__ void prefetch_l2(const void* p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// A stencil value from shared memory.  The face flux asks for a value again in
// each part that uses it.  In FP64 every read stays a read (volatile): merged
// into one, the compiler holds a face's 30 values (60 registers) across the
// whole flux and spills 384 B per thread (to L2: shared memory leaves L1 about
// 20 KB) -- stage 2 at 256x256x128 1.86 ms against 1.64 with 64 B left.
__device__ __forceinline__ double sm_read(const double* p) { return *(const volatile double*)p; }

// PWT: row pitch of the plane buffer (PW; 24 in the FP64 TMA kernel, whose
// plane is one TMA box starting at tile x = -4)
template <int PWT>
struct Smem {
  double ring[6][NEQ][NC];
  double plane[NEQ][PH][PWT];
  double fi[NEQ][TJ][TI + 1];
  double fj[NEQ][TJ + 1][TI];
};

// Face-node area vectors of one plane, staged by the synchronous kernel.
struct AreaSync {
  double sx[3][TJ][TI + 2];  // J*grad(xi) at node (i0-1+c, j0+r)
  double sy[3][TJ + 2][TI];  // J*grad(eta) at node (i0+c, j0-1+r)
};

// TMA staging: the ring column of a plane lands in its ring
// slot (box 16 x 15 x 1 x 5, the slot's [field][row][col] layout), the whole
// plane with its halo in the plane buffer (box 24 x 21 x 1 x 5 from tile x =
// -4, row pitch 24), the face-node area vectors (FP64) here; all single
// buffers, refilled for the next plane once the current plane's flux rounds
// are over, so the copies travel during the RK update.
struct TmaSmem64 {
  alignas(128) double xi[3][TJ][24];      // J*grad(xi), x = i0-4 .. i0+19, rows j0 .. j0+14
  alignas(128) double eta[3][TJ + 2][TI];  // J*grad(eta), x = i0 .. i0+15, rows j0-1 .. j0+15
  alignas(8) unsigned long long bar[2];
};
// bytes of the warm-up set (the ring's first six planes) and of a plane's set
// (its ring column three planes ahead, the plane with halo, the area vectors)
constexpr unsigned kTma64Warm = (unsigned)(6 * sizeof(double) * NEQ * NC);
constexpr unsigned kTma64Plane =
    (unsigned)(sizeof(double) * (NEQ * NC + NEQ * PH * 24 + 3 * TJ * 24 + 3 * (TJ + 2) * TI));

constexpr size_t round_to(size_t x, size_t m) { return (x + m - 1) / m * m; }

// dynamic shared memory: Smem and TmaSmem64 from a 128-byte boundary (TMA), or
// Smem and AreaSync
template <bool TMA>
__host__ __device__ constexpr size_t stage_smem() {
  return TMA ? 128 + round_to(sizeof(Smem<24>), 128) + sizeof(TmaSmem64) : round_to(sizeof(Smem<PW>), 16) + sizeof(AreaSync);
}

// 2 CTAs per SM (shared memory allows no more).  The work of one CTA: tile
// `tile` of the block's (i, j) tiling, k chunk `kc`.  TMA: TMA staging of the
// ring column, plane and area vectors, else synchronous loads.
template <bool VISC, int MODE, bool TMA>
__device__ __forceinline__ void stage_body(const StageCore& a, const StageMaps* tm, int tile, int kc,
                                           unsigned char* smem_raw) {
  using R = double;
  constexpr int PWT = TMA ? 24 : PW;  // plane row pitch
  constexpr int X0 = TMA ? 1 : 0;     // plane column of tile x = -H, minus H
  using SM = Smem<PWT>;
  unsigned char* base =
      TMA ? reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127)) : smem_raw;
  SM& sm = *reinterpret_cast<SM*>(base);
  unsigned char* tail = base + round_to(sizeof(SM), TMA ? 128 : 16);
  TmaSmem64* t64 = reinterpret_cast<TmaSmem64*>(tail);
  AreaSync* asy = reinterpret_cast<AreaSync*>(tail);

  const StepState* st = a.st;
  if (MODE != 0 && st->done) return;
  const double dt = (MODE != 0) ? st->dt : 0.0;

  const Dims& d = a.d;
  const int t = threadIdx.x;
  const int ti0 = 1 + TI * (tile % a.ntile_i);
  const int tj0 = 1 + TJ * (tile / a.ntile_i);
  const int kb = 1 + a.kchunk * kc;
  const int ke = min(kb + a.kchunk, d.KM - 1);
  if (kb >= ke) return;
  const long VOL = d.VOL;
  const FluxConsts<R> C{(R)a.gamma, (R)a.gam1, (R)a.gam1_inv};

  // The i-face (round A) and j-face (round B) of this thread: half-warps take
  // 16 faces of one row each, the two halves of a warp rows 8 apart.  Round A:
  // warps 0-6 take rows w and w+8, faces 0..15; warp 7 row 7 and the fx = 16
  // face of rows 0..14.
  auto face_a = [&](int& fx, int& fy) -> bool {
    const int w = t >> 5, l = t & 31;
    if (w < 7) {
      fx = l & 15;
      fy = w + 8 * (l >> 4);
    } else if (l < 16) {
      fx = l;
      fy = 7;
    } else {
      fx = TI;
      fy = l - 16;
    }
    return fy < TJ;
  };
  auto face_b = [&](int& fx, int& fy) {
    fx = t & 15;
    fy = (t >> 5) + 8 * ((t >> 4) & 1);
  };

  // column owned by this thread
  const int cx = t % TI, cy = t / TI;
  const int ci = ti0 + cx, cj = tj0 + cy;
  const bool col_thread = t < NC;
  const bool col_valid = col_thread && ci <= d.IM - 2 && cj <= d.JM - 2;

  auto load_ring = [&](int kp) {
    if (col_thread) {
      R* dst = &sm.ring[(kp + 6) % 6][0][t];
      if (ci <= d.IM + 1 && cj <= d.JM + 1) {
        const long o = node_off(d, ci, cj, kp);
#pragma unroll
        for (int n = 0; n < NEQ; ++n) dst[n * NC] = __ldg(a.src + n * VOL + o);
      }
    }
  };
  auto load_zeta = [&](int kp, double z[3]) {
    const long o = node_off(d, ci, cj, kp);
#pragma unroll
    for (int m = 0; m < 3; ++m) z[m] = __ldg(a.area[6 + m] + o);
  };

  // k-face between planes kk and kk+1 of this thread's column
  auto k_face = [&](int kk, const double za[3], const double zb[3], R out[5]) {
    const int s0 = (kk - 2 + 6) % 6;
    auto ld = [&](int p, int n) -> R {
      int s = s0 + p;
      s = s >= 6 ? s - 6 : s;
      return sm_read(&sm.ring[s][n][t]);
    };
    face_flux<R>(ld, 0.5 * (za[0] + zb[0]), 0.5 * (za[1] + zb[1]), 0.5 * (za[2] + zb[2]), C, out);
  };

  // halo node e of a plane: tile-relative (x, y)
  auto halo_xy = [&](int e, int& x, int& y) {
    if (e < NHI) {
      const int c6 = e % (2 * H);
      y = e / (2 * H);
      x = c6 < H ? c6 - H : TI + (c6 - H);
    } else {
      const int e2 = e - NHI;
      const int r6 = e2 / TI;
      x = e2 % TI;
      y = r6 < H ? r6 - H : TJ + (r6 - H);
    }
  };
  // TMA kernel: the copies of plane kp's set -- its ring column three
  // planes ahead (kp+3), the plane with its halo, the area vectors -- on
  // barrier q & 1 (q = kp - kb + 1; the warm-up set is q = 0)
  auto issue_set64 = [&](int kp) {
    if constexpr (TMA) {
      if (t == 0) {
        unsigned long long* bar = &t64->bar[(kp - kb + 1) & 1];
        tma::fence_proxy();
        tma::bar_expect(bar, kTma64Plane);
        const int z = kp + NG, y0 = tj0 + NG;
        const int xl = (int)LP + NG + ti0 - 4, xc = (int)LP + NG + ti0;
        tma::load_4d(&sm.ring[(kp + 3) % 6][0][0], &tm->q_a, xc, y0, kp + 3 + NG, 0, bar);
        tma::load_4d(&sm.plane[0][0][0], &tm->q_b, xl, y0 - H, z, 0, bar);
        tma::load_4d(&t64->xi[0][0][0], &tm->xi, xl, y0, z, 0, bar);
        tma::load_4d(&t64->eta[0][0][0], &tm->eta, xc, y0 - 1, z, 3, bar);
      }
    }
  };

  // L2: plane kp's set and what its faces and update read from memory
  auto prefetch_set = [&](int kp) {
    if constexpr (TMA) {
      const int z = kp + NG, y0 = tj0 + NG, xl = (int)LP + NG + ti0 - 4, xc = (int)LP + NG + ti0;
      tma::prefetch_4d(&tm->q_a, xc, y0, z + 3, 0);
      tma::prefetch_4d(&tm->q_b, xl, y0 - H, z, 0);
      tma::prefetch_4d(&tm->xi, xl, y0, z, 0);
      tma::prefetch_4d(&tm->eta, xc, y0 - 1, z, 3);
      tma::prefetch_4d(&tm->zeta, xc, y0, z + 1, 6);
      tma::prefetch_4d(&tm->iJ, xc, y0, z, 0);
      if (MODE >= 1 && !a.q0_is_src) tma::prefetch_4d(&tm->q0, xc, y0, z, 0);
      if (MODE >= 2 && !a.qp_is_src) tma::prefetch_4d(&tm->qp, xc, y0, z, 0);
    }
  };

  if constexpr (TMA) {
    if (t == 0) {
      tma::bar_init(&t64->bar[0]);
      tma::bar_init(&t64->bar[1]);
      tma::fence_init();
    }
    __syncthreads();  // no thread waits on a barrier before it is initialised
  }
  // warm-up: planes kb-3 .. kb+2 and the kb-1/2 face
  bool landed = true;
  if constexpr (TMA) {
    if (t == 0) {
      tma::bar_expect(&t64->bar[0], kTma64Warm);
      for (int kp = kb - 3; kp <= kb + 2; ++kp)
        tma::load_4d(&sm.ring[(kp + 6) % 6][0][0], &tm->q_a, (int)LP + NG + ti0, tj0 + NG, kp + NG, 0, &t64->bar[0]);
    }
  } else {
    for (int kp = kb - 3; kp <= kb + 2; ++kp) load_ring(kp);
  }
  // the column's J*grad(zeta) at planes k and k+1, in FP64 (the stage-3
  // spectral radius uses it exactly)
  double za[3] = {0, 0, 0}, zb[3] = {0, 0, 0};
  if (col_valid) {
    load_zeta(kb - 1, za);
    load_zeta(kb, zb);
  }
  if constexpr (TMA) landed = tma::bar_wait(&t64->bar[0], 0);
  if (__syncthreads_or(!landed)) {
    if (t == 0) {
      atomicExch(&a.st->stage_fail, 1);
      tma::bar_wait(&t64->bar[0], 0);  // bounded: the copies in flight
    }
    return;
  }
  R fkm[5] = {0, 0, 0, 0, 0};
  if (col_valid) k_face(kb - 1, za, zb, fkm);
#pragma unroll
  for (int m = 0; m < 3; ++m) za[m] = zb[m];
  if constexpr (TMA) {
    __syncthreads();  // the warm-up face has read the slot plane kb+3 lands in
    issue_set64(kb);
  }

  double smax = 0.0;  // running spectral-radius max (stage 3, inviscid)
  bool snan = false;
  constexpr bool kSigma = MODE == 3 && !VISC;
  __shared__ int best;  // the largest spectral radius met so far (sigma.cuh)
  if (kSigma && a.sigma && t == 32) best = __float_as_int(sigma_start(st));

  for (int k = kb; k < ke; ++k) {
    if (t == 0 && k + 1 < ke) prefetch_set(k + 1);
    if (col_valid) load_zeta(k + 1, zb);  // consumed in round C
    // viscous kernels ask L2 for the next plane's viscous divergence
    if (VISC && MODE != 0 && col_valid && k + 1 < ke) {
      const long o = node_off(d, ci, cj, k + 1);
#pragma unroll
      for (int n = 0; n < 4; ++n) prefetch_l2(a.dfv[n] + o);
    }
    // plane k's set (TMA kernel) has landed; a wait that runs out on any thread
    // ends the CTA's work, recorded in st->stage_fail
    unsigned long long* wbar = nullptr;
    unsigned wpar = 0;
    if constexpr (TMA) {
      wbar = &t64->bar[(k - kb + 1) & 1];
      wpar = ((k - kb + 1) >> 1) & 1;
      landed = tma::bar_wait(wbar, wpar);
    }
    if (__syncthreads_or(!landed)) {
      if (t == 0) {
        atomicExch(&a.st->stage_fail, 1);
        tma::bar_wait(wbar, wpar);  // bounded: the copies in flight
      }
      return;
    }
    if constexpr (!TMA) load_ring(k + 3);
    // plane k with halo: interior from the ring, halo from global memory
    if constexpr (!TMA) {
      const int sk = k % 6;
      for (int e = t; e < NC; e += NT) {
        const int x = e % TI, y = e / TI;
#pragma unroll
        for (int n = 0; n < NEQ; ++n) sm.plane[n][y + H][x + H] = sm.ring[sk][n][e];
      }
      // halo: 6 columns x TJ rows (i-halo) then 6 rows x TI columns (j-halo)
      for (int e = t; e < NHI + NHJ; e += NT) {
        int x, y;
        halo_xy(e, x, y);
        const int gi = ti0 + x, gj = tj0 + y;
        if (gi <= d.IM + 1 && gj <= d.JM + 1) {
          const long o = node_off(d, gi, gj, k);
#pragma unroll
          for (int n = 0; n < NEQ; ++n) sm.plane[n][y + H][x + H] = __ldg(a.src + n * VOL + o);
        }
      }
      // area vectors of the face nodes of plane k (synchronous kernels)
      for (int e = t; e < NSX + NSY; e += NT) {
        if (e < NSX) {
          const int c = e % (TI + 2), r = e / (TI + 2);
          const int gi = ti0 - 1 + c, gj = tj0 + r;
          if (gi <= d.IM + 1 && gj <= d.JM + 1) {
            const long o = node_off(d, gi, gj, k);
#pragma unroll
            for (int m = 0; m < 3; ++m) asy->sx[m][r][c] = __ldg(a.area[m] + o);
          }
        } else {
          const int e2 = e - NSX;
          const int c = e2 % TI, r = e2 / TI;
          const int gi = ti0 + c, gj = tj0 - 1 + r;
          if (gi <= d.IM + 1 && gj <= d.JM + 1) {
            const long o = node_off(d, gi, gj, k);
#pragma unroll
            for (int m = 0; m < 3; ++m) asy->sy[m][r][c] = __ldg(a.area[3 + m] + o);
          }
        }
      }
    }
    if constexpr (!TMA) __syncthreads();
    // the area vectors of plane k's face nodes: node (i0-1+c, j0+r) and (i0+c, j0-1+r)
    auto ax = [&](int m, int r, int c) -> R {
      if constexpr (TMA) return t64->xi[m][r][c + 3];
      else return asy->sx[m][r][c];
    };
    auto ay = [&](int m, int r, int c) -> R {
      if constexpr (TMA) return t64->eta[m][r][c];
      else return asy->sy[m][r][c];
    };

    R fkp[5];
    // round A: i-faces.  Face fx (0..TI) of row fy lies between tile columns fx-1 and fx.
    int fx, fy;
    if (face_a(fx, fy)) {
      const int ga = ti0 + fx - 1, gj = tj0 + fy;
      if (ga <= d.IM - 2 && gj <= d.JM - 2) {
        auto ld = [&](int p, int n) -> R { return sm_read(&sm.plane[n][fy + H][fx + p + X0]); };
        R f[5];
        face_flux<R>(ld, 0.5 * (ax(0, fy, fx) + ax(0, fy, fx + 1)), 0.5 * (ax(1, fy, fx) + ax(1, fy, fx + 1)),
                     0.5 * (ax(2, fy, fx) + ax(2, fy, fx + 1)), C, f);
#pragma unroll
        for (int n = 0; n < NEQ; ++n) sm.fi[n][fy][fx] = f[n];
      }
    }
    // round B: j-faces.  Face fy (0..TJ) of column fx lies between tile rows fy-1 and fy.
    {
      face_b(fx, fy);
      const int gi = ti0 + fx, ga = tj0 + fy - 1;
      if (gi <= d.IM - 2 && ga <= d.JM - 2) {
        auto ld = [&](int p, int n) -> R { return sm_read(&sm.plane[n][fy + p][fx + H + X0]); };
        R f[5];
        face_flux<R>(ld, 0.5 * (ay(0, fy, fx) + ay(0, fy + 1, fx)), 0.5 * (ay(1, fy, fx) + ay(1, fy + 1, fx)),
                     0.5 * (ay(2, fy, fx) + ay(2, fy + 1, fx)), C, f);
#pragma unroll
        for (int n = 0; n < NEQ; ++n) sm.fj[n][fy][fx] = f[n];
      }
    }
    // round C: the k+1/2 face of this column
    if (col_valid) k_face(k, za, zb, fkp);
    // stage 3's spectral radius: the column's area vectors in FP32 for its
    // bound, before the staging is refilled
    float ar[9];
    if (kSigma && col_valid) {
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        ar[m] = (float)ax(m, cy, cx + 1);
        ar[3 + m] = (float)ay(m, cy + 1, cx);
        ar[6 + m] = (float)za[m];
      }
    }
    __syncthreads();
    // TMA kernel: plane k+1's set travels during the update (it
    // overwrites the plane, the area vectors and plane k-2's ring slot, which
    // the rounds above were the last to read)
    if (TMA && k + 1 < ke) issue_set64(k + 1);

    if (col_valid) {
      const long o = node_off(d, ci, cj, k);
      double df[NEQ];
#pragma unroll
      for (int n = 0; n < NEQ; ++n)
        df[n] = (sm.fi[n][cy][cx + 1] - sm.fi[n][cy][cx]) + (sm.fj[n][cy + 1][cx] - sm.fj[n][cy][cx]) + (fkp[n] - fkm[n]);
      if (VISC) {
        // the viscous flux divergence, formed by visc_div_kernel (visc.cu)
#pragma unroll
        for (int n = 0; n < 4; ++n) df[n + 1] -= __ldg(a.dfv[n] + o);
      }
      const double iJ = __ldg(a.area[9] + o);
      if (MODE == 0) {
        const long r = 5L * ((ci - 1) + (long)(d.IM - 2) * ((cj - 1) + (long)(d.JM - 2) * (k - 1)));
#pragma unroll
        for (int n = 0; n < NEQ; ++n) a.out[r + n] = ml(df[n], iJ);
      } else {
        const int sk = k % 6;
        double q[NEQ];
#pragma unroll
        for (int n = 0; n < NEQ; ++n) {
          // explicit roundings: the variants and the batched form agree to the bit
          const double x = ml(df[n], iJ);
          const long e = n * VOL + o;
          const double qin = sm.ring[sk][n][t];
          const double q0v = MODE == 3 ? a.q0[e] : __ldg(a.q0 + e);
          const double qpv = MODE >= 2 ? __ldg(a.qp + e) : 0.0;
          if (MODE == 1) q[n] = fm(-dt, x, a.q0_is_src ? qin : q0v);
          else if (MODE == 2) q[n] = fm(0.25, fm(-dt, x, a.qp_is_src ? qin : qpv), ml(0.75, q0v));
          else q[n] = third(fm(2.0, fm(-dt, x, a.qp_is_src ? qin : qpv), q0v));
        }
#pragma unroll
        for (int n = 0; n < NEQ; ++n) a.out[n * VOL + o] = q[n];
        if (VISC) {
          const double r = q[0], ir = __drcp_rn(r);
          const double uu = __dmul_rn(q[1], ir), vv = __dmul_rn(q[2], ir), ww = __dmul_rn(q[3], ir);
          const double ke = __fma_rn(ww, ww, __fma_rn(vv, vv, __dmul_rn(uu, uu)));
          const double pp = __dmul_rn(a.gam1, __fma_rn(-__dmul_rn(0.5, r), ke, q[4]));
          if (!a.lean) a.prim[0][o] = r;
          a.prim[1][o] = uu;
          a.prim[2][o] = vv;
          a.prim[3][o] = ww;
          if (!a.lean) a.prim[4][o] = pp;
          a.prim[5][o] = __ddiv_rn(ml(a.gM2, pp), r);
        } else if (kSigma && a.sigma) {
          // in FP64 only where the FP32 bound reaches the largest met so far
          float qf[NEQ], small;
#pragma unroll
          for (int n = 0; n < NEQ; ++n) qf[n] = (float)q[n];
          const float b = sigma_bound(qf, ar, (float)iJ, (float)a.gamma, (float)a.gam1, small);
          if (sigma_reaches(b, small, __int_as_float(*(volatile int*)&best))) {
            double A[9];
#pragma unroll
            for (int m = 0; m < 9; ++m) A[m] = __ldg(a.area[m] + o);
            const double s = sigma_exact(q, A, iJ, a.gamma, a.gam1);
            if (s != s) snan = true;
            smax = fmax(smax, s);
            sigma_found(&best, s);
          }
        }
      }
    }
#pragma unroll
    for (int n = 0; n < NEQ; ++n) fkm[n] = fkp[n];
#pragma unroll
    for (int m = 0; m < 3; ++m) za[m] = zb[m];
  }

  if constexpr (TMA) {
    // every issued copy was waited for: nothing is in flight; retire the
    // barriers so a batched CTA can initialise them again for its next item
    __syncthreads();
    if (t == 0) {
      tma::bar_inval(&t64->bar[0]);
      tma::bar_inval(&t64->bar[1]);
    }
  }
  if (kSigma && a.sigma) {
    // CTA max, one atomic per CTA
    __shared__ double red[NT / 32];
    __shared__ int rnan;
    if (t == 0) rnan = 0;
    double m = smax;
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, s));
    __syncthreads();
    if (snan) rnan = 1;
    if ((t & 31) == 0) red[t >> 5] = m;
    __syncthreads();
    if (t == 0) {
      for (int w = 1; w < NT / 32; ++w) m = fmax(m, red[w]);
      atomic_max_sigma(&a.st->sigma_bits, rnan ? __longlong_as_double(0x7ff8000000000000ll) : m);
    }
  }
}

template <bool VISC, int MODE, bool TMA>
__global__ void __launch_bounds__(NT, 2) stage_kernel(const __grid_constant__ StageArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  stage_body<VISC, MODE, TMA>(a, &a.tm, blockIdx.x, blockIdx.y, smem_raw);
}

// Many blocks in one launch: persistent CTAs take work items (block, tile, k
// chunk) from a queue (one atomic counter); each item's StageArgs are copied
// from the table into shared memory.  Items are numbered block by block, tiles
// fastest, so CTAs of one block work on neighbouring columns together.  Staged
// by TMA: the item's arguments without their tensor maps are what shared memory
// has room for (12 blocks, 2.2 M nodes, 16-plane items: 976 us per stage staged
// synchronously, 604 by TMA, 589 with 8-plane items).
template <bool VISC, int MODE>
__global__ void __launch_bounds__(NT, 2) stage_kernel_batched(const BatchStage b) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ StageCore args;
  __shared__ int item;
  int maps_of = -1;
  for (;;) {
    if (threadIdx.x == 0) item = (int)atomicAdd(b.counter, 1u);
    __syncthreads();
    const int w = item;
    if (w >= b.total) break;
    const int blk = block_of_cta(b.start, b.nblocks, w);
    copy_core(&args, b.args + blk, NT);
    batch_maps(b.args, blk, maps_of);
    __syncthreads();
    const int local = w - __ldg(b.start + blk);
    const int ntiles = args.ntile_i * args.ntile_j;
    stage_body<VISC, MODE, true>(args, &b.args[blk].tm, local % ntiles, local / ntiles, smem_raw);
    __syncthreads();  // args, item and the shared staging are reused by the next item
  }
}

template <bool VISC, int MODE>
cudaError_t launch_batched_t(const BatchStage& b, cudaStream_t s) {
  const int smem = (int)stage_smem<true>();
  const void* f = (const void*)stage_kernel_batched<VISC, MODE>;
  static int grid = 0;
  if (grid == 0) {
    cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    int per_sm = 0, dev = 0, nsm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, NT, smem);
    if (e == cudaSuccess) e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    grid = nsm * (per_sm > 0 ? per_sm : 1);
  }
  const int g = b.total < grid ? b.total : grid;
  if (g <= 0) return cudaSuccess;
  stage_kernel_batched<VISC, MODE><<<g, NT, smem, s>>>(b);
  return cudaGetLastError();
}

template <bool VISC>
cudaError_t launch_batched_v(const BatchStage& b, int mode, cudaStream_t s) {
  switch (mode) {
    case 1: return launch_batched_t<VISC, 1>(b, s);
    case 2: return launch_batched_t<VISC, 2>(b, s);
    default: return launch_batched_t<VISC, 3>(b, s);
  }
}

template <bool VISC, int MODE, bool TMA>
cudaError_t launch_t(const StageArgs& a, cudaStream_t s) {
  dim3 grid(a.ntile_i * a.ntile_j, (a.d.KM - 2 + a.kchunk - 1) / a.kchunk);
  stage_kernel<VISC, MODE, TMA><<<grid, NT, stage_smem<TMA>(), s>>>(a);
  return cudaGetLastError();
}

template <bool VISC, bool TMA>
cudaError_t prepare_v() {
  const void* f[] = {(const void*)stage_kernel<VISC, 0, TMA>, (const void*)stage_kernel<VISC, 1, TMA>,
                     (const void*)stage_kernel<VISC, 2, TMA>, (const void*)stage_kernel<VISC, 3, TMA>};
  return raise_smem(f, 4, stage_smem<TMA>());
}

template <bool VISC, bool TMA>
cudaError_t launch_v(const StageArgs& a, int mode, cudaStream_t s) {
  switch (mode) {
    case 0: return launch_t<VISC, 0, TMA>(a, s);
    case 1: return launch_t<VISC, 1, TMA>(a, s);
    case 2: return launch_t<VISC, 2, TMA>(a, s);
    default: return launch_t<VISC, 3, TMA>(a, s);
  }
}

}  // namespace

cudaError_t raise_smem(const void* const* kernels, int n, size_t bytes) {
  cudaError_t e = cudaSuccess;
  for (int m = 0; m < n && e == cudaSuccess; ++m) {
    e = cudaFuncSetAttribute(kernels[m], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    // the largest carveout, so that as many CTAs as the kernel is built for fit on an SM
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(kernels[m], cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  }
  return e;
}

cudaError_t stage_prepare() {
  static std::mutex m;
  static bool done = false;
  std::lock_guard<std::mutex> lock(m);
  if (done) return cudaSuccess;
  cudaError_t e = prepare_v<false, false>();
  if (e == cudaSuccess) e = prepare_v<false, true>();
  if (e == cudaSuccess) e = prepare_v<true, false>();
  if (e == cudaSuccess) e = prepare_v<true, true>();
  done = e == cudaSuccess;
  return e;
}

void stage_tiles(const Dims& d, int* ntile_i, int* ntile_j) {
  *ntile_i = (d.IM - 2 + TI - 1) / TI;
  *ntile_j = (d.JM - 2 + TJ - 1) / TJ;
}

// FP64: synchronous (variant 0) or TMA staging (variant 1).  FP32 flux: register
// budgets for 2 (variant 0) or 3 CTAs per SM; the hybrid's variant 2 is accepted
// and runs variant 1's kernel (shared memory holds no fourth CTA).
int stage_variants(bool fp32, bool hybrid) { return fp32 && hybrid ? 3 : 2; }

cudaError_t launch_stage_batched(const BatchStage& b, int mode, bool visc, bool fp32, bool hybrid, cudaStream_t s) {
  if (mode < 1 || mode > 3) return cudaErrorInvalidValue;
  if (fp32) return launch_stage32_batched(b, mode, visc, hybrid, s);
  return visc ? launch_batched_v<true>(b, mode, s) : launch_batched_v<false>(b, mode, s);
}

cudaError_t launch_stage(const StageArgs& a, int mode, bool visc, bool fp32, int variant, cudaStream_t s) {
  if (fp32) return launch_stage32(a, mode, visc, variant, s);
  if (visc) return variant == 1 ? launch_v<true, true>(a, mode, s) : launch_v<true, false>(a, mode, s);
  return variant == 1 ? launch_v<false, true>(a, mode, s) : launch_v<false, false>(a, mode, s);
}

}  // namespace cbns
