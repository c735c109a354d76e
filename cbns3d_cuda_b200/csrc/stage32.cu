// stage32.cu - one SSP-RK3 stage in one kernel with the flux in FP32 (the split
// and hybrid precisions); the FP64 kernel and the work it replaces in the
// reference are described in stage.cu.
//
// Source.  Each state buffer has an FP32 copy beside it, written by whatever
// writes the state (this kernel, the boundary kernels, the uploads), so a
// plane's stencil values arrive in shared memory by TMA as the flux uses them:
// no thread loads, converts or stores a stencil value.  (Converting the FP64
// state on the way in took a third of the kernel's instructions: the ring
// column through registers, the halo boxes through shared memory, the plane's
// copy out of the ring.)  The copies cost 20 B per node and stage in writes and
// save 20 in reads.
// Tiling (2.5D).  A CTA of 128 threads owns a 16 x 15 column of interior nodes
// and marches it through a chunk of k planes.  Shared memory, all written by
// TMA from one elected thread:
//   ring   : the column's state on the 6 planes k-2 .. k+3 (stencil of the k
//            faces), one new plane per step;
//   plane  : plane k, x from -4 to 19 and y from -3 to 17 of the tile (stencils
//            of the i and j faces);
//   areas  : J*grad(xi) and J*grad(eta) at the face nodes of plane k,
//            J*grad(zeta) of planes k and k+1.
// Two faces per thread and round, as packed FP32 pairs (F2, face_flux.cuh):
//   round A: the i-faces of two neighbouring rows (the half-warps' rows 2
//            apart, so a plane row's reads, pitch 24, start 16 banks apart);
//            the sixteenth row's place takes the 17th face of every row;
//   round B: the j-faces likewise;
//   round C: the k+1/2 faces of columns t and t+128 (conflict-free in the ring).
// One packed operation serves two faces: the WENO5 flux issues half the FP32
// instructions.  Face fluxes go to shared memory (two buffers, so a plane has
// one CTA barrier), the k-1/2 fluxes are carried in registers.  After the
// barrier the copies of the next plane are issued and travel during the
// update, their L2 lines and those of the update's operands asked for a plane
// ahead (cp.async.bulk.prefetch.tensor).
// Bound by the FP32 pipe and issue (WENO5) and by load latency (linear faces:
// issue 46%, 3.7 TB/s of DRAM traffic).  Measured against one face per thread
// (256 threads, the FP64 state converted on the way in), us per launch of
// stages 1 / 2 / 3: hybrid 256x256x128 517 / 567 / 617 -> 385 / 446 / 584 (half
// the instructions: 86 M warp instructions for 3.4 M nodes instead of 164 M);
// split 193x161x129 464 / 480 / 519 -> 411 / 422 / 501; 64 viscous hybrid
// blocks 1250 / 1418 / 1327 -> 954 / 1045 / 1009.  Since then the bounded
// spectral radius (sigma.cuh) took from stage 3 and the wider range of the FP32
// weights (face_flux.cuh) added to the split: 387 / 440 / 469, 423 / 443 / 493
// and 861 / 919 / 932.
//
// Hybrid (HYB): each face's sensor decision selects the linear upwind-5 flux,
// evaluated here, or the characteristic WENO5 flux, evaluated before this
// kernel by the WENO5-face pass (weno_faces.cu) and read from its face array.
// The decisions of plane k+1 are read while plane k is computed, and the WENO5
// fluxes of plane k are asked into L1 at its start.
#include <mutex>

#include "cbns_common.cuh"
#include "face_flux.cuh"
#include "sigma.cuh"
#include "stage.cuh"
#include "tma.cuh"

namespace cbns {

namespace {

constexpr int TI = STAGE_TI, TJ = STAGE_TJ, H = 3;
constexpr int NT = 128, NC = TI * TJ;
constexpr int PWX = 24, PH = TJ + 2 * H;
constexpr int SLOT = 1216;                // floats of a ring slot: 5 x 240, padded to 128 bytes
constexpr int ZS = 736;                   // floats of a zeta plane: 3 x 240, padded to 128 bytes
static_assert(TI == 16 && TJ == 15, "face mapping of the rounds");
static_assert((NEQ - 1) * NC + NT + NT <= SLOT, "column t + 128 stays inside the slot");

struct alignas(128) Smem32 {
  float ring[6][SLOT];
  alignas(128) float plane[NEQ][PH][PWX];
  alignas(128) float xi[3][TJ][PWX];       // x = -4 .. 19
  alignas(128) float eta[3][TJ + 2][TI];   // rows -1 .. 15
  alignas(128) float zt[2][ZS];            // plane p in zt[p & 1]
  float fi[2][NEQ][TJ][TI + 1];            // plane p in buffer p & 1
  float fj[2][NEQ][TJ + 1][TI];
  alignas(8) unsigned long long bar[2];
  int best;  // the largest spectral radius met so far (sigma.cuh)
};
constexpr size_t kSmem = sizeof(Smem32) + 128;
// transaction bytes: a plane's set, the warm-up set (six ring planes, two zeta planes)
constexpr unsigned kSet = 4u * (NEQ * NC + NEQ * PH * PWX + 3 * TJ * PWX + 3 * (TJ + 2) * TI + 3 * NC);
constexpr unsigned kWarm = 4u * (6 * NEQ * NC + 2 * 3 * NC);

__device__ __forceinline__ void prefetch_l1(const void* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

// The work of one CTA: tile `tile` of the block's (i, j) tiling, k chunk `kc`.
template <bool VISC, int MODE, bool HYB>
__device__ __forceinline__ void stage32_body(const StageCore& a, const StageMaps* tm, int tile, int kc,
                                             unsigned char* smem_raw) {
  Smem32& sm = *reinterpret_cast<Smem32*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
  const StepState* st = a.st;
  if (MODE != 0 && st->done) return;
  const double dt = (MODE != 0) ? st->dt : 0.0;
  const Dims& d = a.d;
  const int t = threadIdx.x;
  const int ti0 = 1 + TI * (tile % a.ntile_i), tj0 = 1 + TJ * (tile / a.ntile_i);
  const int kb = 1 + a.kchunk * kc, ke = min(kb + a.kchunk, d.KM - 1);
  if (kb >= ke) return;
  const long VOL = d.VOL;
  const FluxConsts<float> C{(float)a.gamma, (float)a.gam1, (float)a.gam1_inv};

  // TMA copies (thread 0 only).  x coordinates: LP + NG + ti0 is a multiple of
  // 16 elements, so every box starts on a 16-byte boundary.
  const int xc = (int)LP + NG + ti0, y0 = tj0 + NG;
  auto slot = [&](int kp) -> float* { return sm.ring[(kp + 6) % 6]; };
  auto issue_ring_zeta = [&](int kp, unsigned long long* bar) {  // ring plane kp+3, zeta plane kp+1
    tma::load_4d(slot(kp + 3), &tm->q_a, xc, y0, kp + 3 + NG, 0, bar);
    tma::load_4d(sm.zt[(kp + 1) & 1], &tm->zeta, xc, y0, kp + 1 + NG, 6, bar);
  };
  auto issue_plane = [&](int kp, unsigned long long* bar) {
    const int z = kp + NG;
    tma::load_4d(sm.plane, &tm->q_b, xc - 4, y0 - H, z, 0, bar);
    tma::load_4d(sm.xi, &tm->xi, xc - 4, y0, z, 0, bar);
    tma::load_4d(sm.eta, &tm->eta, xc, y0 - 1, z, 3, bar);
  };
  auto prefetch_set = [&](int kp) {  // L2: plane kp's set and its update's operands
    const int z = kp + NG;
    tma::prefetch_4d(&tm->q_a, xc, y0, kp + 3 + NG, 0);
    tma::prefetch_4d(&tm->q_b, xc - 4, y0 - H, z, 0);
    tma::prefetch_4d(&tm->xi, xc - 4, y0, z, 0);
    tma::prefetch_4d(&tm->eta, xc, y0 - 1, z, 3);
    tma::prefetch_4d(&tm->zeta, xc, y0, z + 1, 6);
    if (MODE != 0) {
      tma::prefetch_4d(&tm->iJ, xc, y0, z, 0);
      tma::prefetch_4d(&tm->q0, xc, y0, z, 0);
      if (MODE >= 2) tma::prefetch_4d(&tm->qp, xc, y0, z, 0);
      if (VISC) tma::prefetch_4d(&tm->dfv, xc, y0, z, 0);
    }
  };

  constexpr bool kSigma = MODE == 3 && !VISC;
  if (kSigma && a.sigma && t == 32) sm.best = __float_as_int(sigma_start(st));
  if (t == 0) {
    tma::bar_init(&sm.bar[0]);
    tma::bar_init(&sm.bar[1]);
    tma::fence_init();
    // warm-up: planes kb-3 .. kb+2 and the zeta planes of the kb-1/2 face; then
    // what plane kb's set can bring before that face is done
    tma::bar_expect(&sm.bar[0], kWarm);
    for (int kp = kb - 3; kp <= kb + 2; ++kp) tma::load_4d(slot(kp), &tm->q_a, xc, y0, kp + NG, 0, &sm.bar[0]);
    tma::load_4d(sm.zt[(kb - 1) & 1], &tm->zeta, xc, y0, kb - 1 + NG, 6, &sm.bar[0]);
    tma::load_4d(sm.zt[kb & 1], &tm->zeta, xc, y0, kb + NG, 6, &sm.bar[0]);
    tma::bar_expect(&sm.bar[1], kSet);
    issue_plane(kb, &sm.bar[1]);
    tma::prefetch_4d(&tm->q_a, xc, y0, kb + 3 + NG, 0);
    tma::prefetch_4d(&tm->zeta, xc, y0, kb + 1 + NG, 6);
  }

  // the thread's faces and columns
  const int c = t & 15, h = (t >> 4) & 1, r0 = 4 * (t >> 5) + 2 * h, r1 = r0 + 1;
  const bool last = r1 == TJ;  // this row's place: the 17th face of row c
  const int ax1 = last ? TI : c, ay1 = last ? c : r1;
  const bool vA0 = ti0 + c - 1 <= d.IM - 2 && tj0 + r0 <= d.JM - 2;
  const bool vA1 = ay1 < TJ && ti0 + ax1 - 1 <= d.IM - 2 && tj0 + ay1 <= d.JM - 2;
  const bool vB0 = ti0 + c <= d.IM - 2 && tj0 + r0 - 1 <= d.JM - 2;
  const bool vB1 = ti0 + c <= d.IM - 2 && tj0 + r1 - 1 <= d.JM - 2;
  const int cy0 = t >> 4, cy1 = cy0 + 8;
  const int ci = ti0 + c, cj0 = tj0 + cy0, cj1 = tj0 + cy1;
  const bool vC0 = ci <= d.IM - 2 && cj0 <= d.JM - 2;
  const bool vC1 = cy1 < TJ && ci <= d.IM - 2 && cj1 <= d.JM - 2;

  // Hybrid: decisions (global face index: i-faces, j-faces, k-faces in the
  // reference's Ep/Fp/Gp order; 32-bit, checked in cbns_create): 0 = linear
  // upwind-5, evaluated here; 1 = characteristic WENO5, evaluated ahead into
  // a.wflux.  While the audit has set force_weno every face is a WENO5 face.
  const bool all_weno = HYB && st->force_weno;
  int eA0 = 0, eA1 = 0, eB0 = 0, eB1 = 0, eC0 = 0, eC1 = 0, sA = 0, sB = 0, sC = 0;
  if constexpr (HYB) {
    const int nfi = (d.IM - 1) * (d.JM - 2) * (d.KM - 2), nfj = (d.IM - 2) * (d.JM - 1) * (d.KM - 2);
    sA = (d.IM - 1) * (d.JM - 2);
    sB = (d.IM - 2) * (d.JM - 1);
    sC = (d.IM - 2) * (d.JM - 2);
    eA0 = (ti0 + c - 1) + (d.IM - 1) * (tj0 + r0 - 1) - sA;  // + k * stride
    eA1 = (ti0 + ax1 - 1) + (d.IM - 1) * (tj0 + ay1 - 1) - sA;
    eB0 = nfi + (ci - 1) + (d.IM - 2) * (tj0 + r0 - 1) - sB;
    eB1 = nfi + (ci - 1) + (d.IM - 2) * (tj0 + r1 - 1) - sB;
    eC0 = nfi + nfj + (ci - 1) + (d.IM - 2) * (cj0 - 1);
    eC1 = nfi + nfj + (ci - 1) + (d.IM - 2) * (cj1 - 1);
  }
  // the decision bytes of the thread's faces of plane k, as loaded: combined
  // into bits only when plane k is reached, so no thread waits for them
  auto load_mask = [&](int k, unsigned char m[6]) {
    if constexpr (HYB) {
      if (all_weno) return;
      if (vA0) m[0] = __ldg(a.mask + (eA0 + k * sA));
      if (vA1) m[1] = __ldg(a.mask + (eA1 + k * sA));
      if (vB0) m[2] = __ldg(a.mask + (eB0 + k * sB));
      if (vB1) m[3] = __ldg(a.mask + (eB1 + k * sB));
      if (vC0) m[4] = __ldg(a.mask + (eC0 + k * sC));
      if (vC1) m[5] = __ldg(a.mask + (eC1 + k * sC));
    }
  };
  auto mask_bits = [&](const unsigned char m[6]) -> unsigned {
    if (all_weno) return 0x3fu;
    unsigned r = 0;
#pragma unroll
    for (int n = 0; n < 6; ++n) r |= (unsigned)(m[n] != 0) << n;
    return r;
  };
  auto prefetch_weno = [&](int k, unsigned m) {
    if ((m & 1u) && vA0) prefetch_l1(a.wflux + 8l * (eA0 + k * sA));
    if ((m & 2u) && vA1) prefetch_l1(a.wflux + 8l * (eA1 + k * sA));
    if ((m & 4u) && vB0) prefetch_l1(a.wflux + 8l * (eB0 + k * sB));
    if ((m & 8u) && vB1) prefetch_l1(a.wflux + 8l * (eB1 + k * sB));
    if ((m & 16u) && vC0) prefetch_l1(a.wflux + 8l * (eC0 + k * sC));
    if ((m & 32u) && vC1) prefetch_l1(a.wflux + 8l * (eC1 + k * sC));
  };
  // the fluxes of two faces: ld the pair's stencil, n its area vectors, m2 its
  // decisions (bit 0: first), e0/e1 its face indices, v0/v1 whether they exist
  auto flux = [&](const auto& ld, F2 nx, F2 ny, F2 nz, unsigned m2, int e0, int e1, bool v0, bool v1, F2 out[5]) {
    if constexpr (HYB) {
      if (m2 != 3u) face_flux_linear<F2>(ld, nx, ny, nz, C, out);
      if (m2) {
        float f0[5] = {0.f, 0.f, 0.f, 0.f, 0.f}, f1[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
        if (m2 != 3u)
          for (int n = 0; n < NEQ; ++n) halves(out[n], f0[n], f1[n]);
        auto get = [&](int e, float f[5]) {
          const float* w = a.wflux + 8l * e;
          const float4 v = __ldg(reinterpret_cast<const float4*>(w));
          f[0] = v.x;
          f[1] = v.y;
          f[2] = v.z;
          f[3] = v.w;
          f[4] = __ldg(w + 4);
        };
        if ((m2 & 1u) && v0) get(e0, f0);
        if ((m2 & 2u) && v1) get(e1, f1);
#pragma unroll
        for (int n = 0; n < NEQ; ++n) out[n] = mk(f0[n], f1[n]);
      }
    } else {
      face_flux<F2>(ld, nx, ny, nz, C, out);
    }
  };
  const F2 half = cst<F2>(0.5);
  // the k-faces between planes kk and kk+1 of the thread's columns
  auto k_face = [&](int kk, unsigned m2, F2 out[5]) {
    int so[6];
    so[0] = ((kk + 4) % 6) * SLOT + t;
#pragma unroll
    for (int p = 1; p < 6; ++p) so[p] = so[p - 1] >= 5 * SLOT ? so[p - 1] - 5 * SLOT : so[p - 1] + SLOT;
    const float* ring = &sm.ring[0][0];
    auto ld = [&](int p, int n) -> F2 { return mk(ring[so[p] + n * NC], ring[so[p] + n * NC + NT]); };
    const float *za = sm.zt[kk & 1] + t, *zb = sm.zt[(kk + 1) & 1] + t;
    auto nv = [&](int m) -> F2 {
      return ml(half, ad(mk(za[m * NC], za[m * NC + NT]), mk(zb[m * NC], zb[m * NC + NT])));
    };
    flux(ld, nv(0), nv(1), nv(2), m2, eC0 + kk * sC, eC1 + kk * sC, vC0, vC1, out);
  };

  __syncthreads();  // no thread waits on a barrier before it is initialised
  const unsigned mwarm = (HYB && !all_weno)
                             ? (unsigned)(vC0 && __ldg(a.mask + (eC0 + (kb - 1) * sC)) != 0) |
                                   (unsigned)(vC1 && __ldg(a.mask + (eC1 + (kb - 1) * sC)) != 0) << 1
                             : 3u;
  unsigned char mraw[6] = {1, 1, 1, 1, 1, 1};  // 1: no second flux for a face that does not exist
  load_mask(kb, mraw);
  bool landed = tma::bar_wait(&sm.bar[0], 0);
  F2 fkm[5];
  k_face(kb - 1, mwarm, fkm);
  if (__syncthreads_or(!landed)) {
    if (t == 0) {
      atomicExch(&a.st->stage_fail, 1);
      tma::bar_wait(&sm.bar[0], 0);  // bounded: the copies in flight
      // bar[1] still waits for the copies issue_ring_zeta would have brought;
      // the plane's copies were issued before and are given the same time
      tma::bar_wait(&sm.bar[1], 0);
    }
    return;
  }
  if (t == 0) {
    tma::fence_proxy();
    issue_ring_zeta(kb, &sm.bar[1]);  // the slots the warm-up face has read
  }

  double smax = 0.0;  // running spectral-radius max (stage 3, inviscid)
  bool snan = false;

  for (int k = kb; k < ke; ++k) {
    const unsigned mcur = HYB ? mask_bits(mraw) : 0u;
    if (t == 0 && k + 1 < ke) prefetch_set(k + 1);
    if constexpr (HYB) {
      prefetch_weno(k, mcur);
      if (k + 1 < ke) load_mask(k + 1, mraw);
    }
    unsigned long long* bar = &sm.bar[(k - kb + 1) & 1];
    const unsigned par = ((unsigned)(k - kb + 1) >> 1) & 1u;
    landed = tma::bar_wait(bar, par);
    float(*fi)[TJ][TI + 1] = sm.fi[k & 1];
    float(*fj)[TJ + 1][TI] = sm.fj[k & 1];
    F2 f[5];
    // round A: face x of row y lies between tile columns x-1 and x
    {
      const float *p0 = &sm.plane[0][r0 + H][c + 1], *p1 = &sm.plane[0][ay1 + H][ax1 + 1];
      auto ld = [&](int p, int n) -> F2 { return mk(p0[n * PH * PWX + p], p1[n * PH * PWX + p]); };
      const float *a0 = &sm.xi[0][r0][c + 3], *a1 = &sm.xi[0][ay1][ax1 + 3];
      auto nv = [&](int m) -> F2 {
        return ml(half, ad(mk(a0[m * TJ * PWX], a1[m * TJ * PWX]), mk(a0[m * TJ * PWX + 1], a1[m * TJ * PWX + 1])));
      };
      flux(ld, nv(0), nv(1), nv(2), mcur & 3u, eA0 + k * sA, eA1 + k * sA, vA0, vA1, f);
#pragma unroll
      for (int n = 0; n < NEQ; ++n) {
        float x, y;
        halves(f[n], x, y);
        fi[n][r0][c] = x;
        if (ay1 < TJ) fi[n][ay1][ax1] = y;
      }
    }
    // round B: face y of column x lies between tile rows y-1 and y
    {
      const float* p0 = &sm.plane[0][r0][c + 4];
      auto ld = [&](int p, int n) -> F2 { return mk(p0[n * PH * PWX + p * PWX], p0[n * PH * PWX + (p + 1) * PWX]); };
      const float* a0 = &sm.eta[0][r0][c];
      auto nv = [&](int m) -> F2 {
        const float* q = a0 + m * (TJ + 2) * TI;
        return ml(half, ad(mk(q[0], q[TI]), mk(q[TI], q[2 * TI])));
      };
      flux(ld, nv(0), nv(1), nv(2), (mcur >> 2) & 3u, eB0 + k * sB, eB1 + k * sB, vB0, vB1, f);
#pragma unroll
      for (int n = 0; n < NEQ; ++n) {
        float x, y;
        halves(f[n], x, y);
        fj[n][r0][c] = x;
        fj[n][r1][c] = y;
      }
    }
    // the update's operands: the hybrid, whose linear flux leaves the
    // registers, loads both columns' before round C, so that they travel during
    // it; with the WENO5 flux each column's in its update (loaded ahead they
    // spill)
    const long o0 = node_off(d, ci, cj0, k), o1 = node_off(d, ci, cj1, k);
    double iJ[2] = {0.0, 0.0}, q0v[2][NEQ], qpv[2][NEQ];
    auto load_operands = [&](int q2) {
      if (!(q2 ? vC1 : vC0)) return;
      const long o = q2 ? o1 : o0;
      iJ[q2] = __ldg(a.area[9] + o);
      if (MODE == 0) return;
#pragma unroll
      for (int n = 0; n < NEQ; ++n) {
        q0v[q2][n] = MODE == 3 ? a.q0[n * VOL + o] : __ldg(a.q0 + n * VOL + o);
        if (MODE >= 2) qpv[q2][n] = __ldg(a.qp + n * VOL + o);
      }
    };
    if (HYB) {
      load_operands(0);
      load_operands(1);
    }
    // round C: the k+1/2 faces of the thread's columns
    F2 fkp[5];
    k_face(k, (mcur >> 4) & 3u, fkp);
    // stage 3's spectral radius: the columns' area vectors, whose buffers are
    // refilled during the update
    F2 ar[9];
    if (kSigma) {
      const int y1 = min(cy1, TJ - 1);
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        ar[m] = mk(sm.xi[m][cy0][c + 4], sm.xi[m][y1][c + 4]);
        ar[3 + m] = mk(sm.eta[m][cy0 + 1][c], sm.eta[m][y1 + 1][c]);
        ar[6 + m] = mk(sm.zt[k & 1][m * NC + t], sm.zt[k & 1][m * NC + y1 * TI + c]);
      }
    }
    if (__syncthreads_or(!landed)) {
      if (t == 0) {
        atomicExch(&a.st->stage_fail, 1);
        tma::bar_wait(bar, par);  // bounded: the copies in flight
      }
      return;
    }
    // plane k+1's set travels during the update (the rounds above were the
    // last to read what it overwrites)
    if (t == 0 && k + 1 < ke) {
      unsigned long long* nb = &sm.bar[(k - kb + 2) & 1];
      tma::fence_proxy();
      tma::bar_expect(nb, kSet);
      issue_plane(k + 1, nb);
      issue_ring_zeta(k + 1, nb);
    }
    // the update of the two columns
    float qf[2][NEQ] = {{1.f, 0.f, 0.f, 0.f, 0.f}, {1.f, 0.f, 0.f, 0.f, 0.f}};
    float fk[2][5];
#pragma unroll
    for (int n = 0; n < NEQ; ++n) halves(sb(fkp[n], fkm[n]), fk[0][n], fk[1][n]);
#pragma unroll
    for (int q2 = 0; q2 < 2; ++q2) {
      const int cy = q2 ? cy1 : cy0, cj = q2 ? cj1 : cj0;
      if (!(q2 ? vC1 : vC0)) continue;
      if (!HYB) load_operands(q2);
      const long o = q2 ? o1 : o0;
      double df[NEQ];
#pragma unroll
      for (int n = 0; n < NEQ; ++n)
        df[n] = (double)(fi[n][cy][c + 1] - fi[n][cy][c]) + (double)(fj[n][cy + 1][c] - fj[n][cy][c]) +
                (double)fk[q2][n];
      if (VISC) {
        // the viscous flux divergence, formed by visc_div_kernel (visc.cu)
#pragma unroll
        for (int n = 0; n < 4; ++n) df[n + 1] -= (double)__ldg(reinterpret_cast<const float*>(a.dfv[n]) + o);
      }
      if (MODE == 0) {
        const long r = 5L * ((ci - 1) + (long)(d.IM - 2) * ((cj - 1) + (long)(d.JM - 2) * (k - 1)));
#pragma unroll
        for (int n = 0; n < NEQ; ++n) a.out[r + n] = df[n] * iJ[q2];
      } else {
        double q[NEQ];
#pragma unroll
        for (int n = 0; n < NEQ; ++n) {
          const double L = dt * (df[n] * iJ[q2]);
          if (MODE == 1) q[n] = q0v[q2][n] - L;
          else if (MODE == 2) q[n] = 0.75 * q0v[q2][n] + 0.25 * (qpv[q2][n] - L);
          else q[n] = (q0v[q2][n] + 2.0 * (qpv[q2][n] - L)) * (1.0 / 3.0);  // one ulp from the plain kernel's division
        }
#pragma unroll
        for (int n = 0; n < NEQ; ++n) {
          a.out[n * VOL + o] = q[n];
          a.out32[n * VOL + o] = qf[q2][n] = (float)q[n];
        }
        if (VISC) {
          const double r = q[0], ir = __drcp_rn(r);
          const double uu = __dmul_rn(q[1], ir), vv = __dmul_rn(q[2], ir), ww = __dmul_rn(q[3], ir);
          const double kk = __fma_rn(ww, ww, __fma_rn(vv, vv, __dmul_rn(uu, uu)));
          const double pp = __dmul_rn(a.gam1, __fma_rn(-__dmul_rn(0.5, r), kk, q[4]));
          if (!a.lean) a.prim[0][o] = r;
          a.prim[1][o] = uu;
          a.prim[2][o] = vv;
          a.prim[3][o] = ww;
          if (!a.lean) a.prim[4][o] = pp;
          a.prim[5][o] = __ddiv_rn(ml(a.gM2, pp), r);
        }
      }
    }
    // stage 3: the columns whose FP32 bound reaches the largest spectral radius
    // met so far are evaluated in FP64, from the FP32 copies of the xi and eta
    // vectors (as the fluxes use them; dt moves by ~1e-7 relative) and the FP64
    // zeta vectors
    if (kSigma && a.sigma) {
      F2 qb[NEQ], small;
#pragma unroll
      for (int n = 0; n < NEQ; ++n) qb[n] = mk(qf[0][n], qf[1][n]);
      float b[2], sl[2];
      const F2 bound = sigma_bound(qb, ar, mk((float)iJ[0], (float)iJ[1]), C.gamma, C.gam1, small);
      halves(bound, b[0], b[1]);
      halves(small, sl[0], sl[1]);
      const float found = __int_as_float(*(volatile int*)&sm.best);
#pragma unroll 1
      for (int q2 = 0; q2 < 2; ++q2) {
        if (!(q2 ? vC1 : vC0) || !sigma_reaches(q2 ? b[1] : b[0], q2 ? sl[1] : sl[0], found)) continue;
        const long o = q2 ? o1 : o0;
        double q[NEQ], A[9];
#pragma unroll
        for (int n = 0; n < NEQ; ++n) q[n] = a.out[n * VOL + o];
#pragma unroll
        for (int m = 0; m < 6; ++m) A[m] = (double)__ldg(a.area32[m] + o);
#pragma unroll
        for (int m = 6; m < 9; ++m) A[m] = __ldg(a.area[m] + o);
        const double s = sigma_exact(q, A, __ldg(a.area[9] + o), a.gamma, a.gam1);
        if (s != s) snan = true;
        smax = fmax(smax, s);
        sigma_found(&sm.best, s);
      }
    }
#pragma unroll
    for (int n = 0; n < NEQ; ++n) fkm[n] = fkp[n];
  }

  // every issued copy was waited for: nothing is in flight; retire the
  // barriers so a batched CTA can initialise them again for its next item
  __syncthreads();
  if (t == 0) {
    tma::bar_inval(&sm.bar[0]);
    tma::bar_inval(&sm.bar[1]);
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

template <bool VISC, int MODE, bool HYB, int NB>
__global__ void __launch_bounds__(NT, NB) stage32_kernel(const __grid_constant__ StageArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  stage32_body<VISC, MODE, HYB>(a, &a.tm, blockIdx.x, blockIdx.y, smem_raw);
}

// Many blocks in one launch, as stage_kernel_batched (stage.cu).
template <bool VISC, int MODE, bool HYB>
__global__ void __launch_bounds__(NT, 3) stage32_kernel_batched(const BatchStage b) {
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
    stage32_body<VISC, MODE, HYB>(args, &b.args[blk].tm, local % ntiles, local / ntiles, smem_raw);
    __syncthreads();  // args, item and the shared staging are reused by the next item
  }
}

template <bool VISC, int MODE, bool HYB>
cudaError_t launch_batched_t(const BatchStage& b, cudaStream_t s) {
  const void* f = (const void*)stage32_kernel_batched<VISC, MODE, HYB>;
  static int grid = 0;
  if (grid == 0) {
    cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    int per_sm = 0, dev = 0, nsm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, NT, kSmem);
    if (e == cudaSuccess) e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    grid = nsm * (per_sm > 0 ? per_sm : 1);
  }
  const int g = b.total < grid ? b.total : grid;
  if (g <= 0) return cudaSuccess;
  stage32_kernel_batched<VISC, MODE, HYB><<<g, NT, kSmem, s>>>(b);
  return cudaGetLastError();
}

template <bool VISC, bool HYB>
cudaError_t launch_batched_v(const BatchStage& b, int mode, cudaStream_t s) {
  switch (mode) {
    case 1: return launch_batched_t<VISC, 1, HYB>(b, s);
    case 2: return launch_batched_t<VISC, 2, HYB>(b, s);
    default: return launch_batched_t<VISC, 3, HYB>(b, s);
  }
}

template <bool VISC, int MODE, bool HYB, int NB>
cudaError_t launch_t(const StageArgs& a, cudaStream_t s) {
  dim3 grid(a.ntile_i * a.ntile_j, (a.d.KM - 2 + a.kchunk - 1) / a.kchunk);
  stage32_kernel<VISC, MODE, HYB, NB><<<grid, NT, kSmem, s>>>(a);
  return cudaGetLastError();
}

template <bool VISC, bool HYB, int NB>
cudaError_t launch_v(const StageArgs& a, int mode, cudaStream_t s) {
  switch (mode) {
    case 0: return launch_t<VISC, 0, HYB, NB>(a, s);
    case 1: return launch_t<VISC, 1, HYB, NB>(a, s);
    case 2: return launch_t<VISC, 2, HYB, NB>(a, s);
    default: return launch_t<VISC, 3, HYB, NB>(a, s);
  }
}

template <bool HYB, int NB>
cudaError_t launch_h(const StageArgs& a, int mode, bool visc, cudaStream_t s) {
  return visc ? launch_v<true, HYB, NB>(a, mode, s) : launch_v<false, HYB, NB>(a, mode, s);
}

template <bool VISC, bool HYB, int NB>
cudaError_t prepare_v() {
  const void* f[] = {(const void*)stage32_kernel<VISC, 0, HYB, NB>, (const void*)stage32_kernel<VISC, 1, HYB, NB>,
                     (const void*)stage32_kernel<VISC, 2, HYB, NB>, (const void*)stage32_kernel<VISC, 3, HYB, NB>};
  return raise_smem(f, 4, kSmem);
}

template <int NB>
cudaError_t prepare_nb() {
  cudaError_t e = prepare_v<false, false, NB>();
  if (e == cudaSuccess) e = prepare_v<false, true, NB>();
  if (e == cudaSuccess) e = prepare_v<true, false, NB>();
  if (e == cudaSuccess) e = prepare_v<true, true, NB>();
  return e;
}

}  // namespace

cudaError_t stage32_prepare() {
  static std::mutex m;
  static bool done = false;
  std::lock_guard<std::mutex> lock(m);
  if (done) return cudaSuccess;
  cudaError_t e = prepare_nb<2>();
  if (e == cudaSuccess) e = prepare_nb<3>();
  done = e == cudaSuccess;
  return e;
}

cudaError_t launch_stage32(const StageArgs& a, int mode, bool visc, int variant, cudaStream_t s) {
  if (a.mask) return variant == 0 ? launch_h<true, 2>(a, mode, visc, s) : launch_h<true, 3>(a, mode, visc, s);
  return variant == 0 ? launch_h<false, 2>(a, mode, visc, s) : launch_h<false, 3>(a, mode, visc, s);
}

cudaError_t launch_stage32_batched(const BatchStage& b, int mode, bool visc, bool hybrid, cudaStream_t s) {
  if (visc) return hybrid ? launch_batched_v<true, true>(b, mode, s) : launch_batched_v<true, false>(b, mode, s);
  return hybrid ? launch_batched_v<false, true>(b, mode, s) : launch_batched_v<false, false>(b, mode, s);
}

}  // namespace cbns
