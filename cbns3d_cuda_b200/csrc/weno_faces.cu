// weno_faces.cu - the WENO5 faces of a hybrid stage, evaluated ahead of the
// stage kernel.
//
// The learned sensor sends about one face in eight to the characteristic
// WENO5 flux (the reference's rec_riemann kernels, src/rec_riemann_kernel.cu,
// called from calc_numerical_flux, src/calc_numerical_flux.cu:15-74) and the
// rest to the linear upwind-5 flux.  Evaluating both inside the stage kernel
// gives the whole stage kernel the register budget and the control flow of
// WENO5 while most of its work is linear.  So, per step, the faces whose
// decision is set are listed once, by the last widening pass, and per stage this
// pass evaluates the listed faces into a face array (8 floats per face, 5
// used: one 16-byte and one 4-byte access), where the stage kernel, which
// holds only the linear flux, reads them.  While force_weno is set (the audit
// rejected the step's decisions, or the sensor timed out) the pass evaluates
// every face.
//
// Stencils are read from the stage input's FP32 copy, as the stage kernel reads
// them, and the face normals are formed from the same FP32 area vectors, so a
// face gets the flux the stage kernel would compute for it.
#include "cbns_common.cuh"
#include "face_flux.cuh"
#include "sensor_kernels.cuh"
#include "stage.cuh"

namespace cbns {

namespace {

constexpr int WT = 128;       // evaluation kernel: threads

// The faces of one kind: the first face index and the count (i-faces, then
// j-faces, then k-faces in the global face numbering).
__host__ __device__ __forceinline__ void kind_range(const Dims& d, int kind, long* first, long* count) {
  const long nfi = (long)(d.IM - 1) * (d.JM - 2) * (d.KM - 2);
  const long nfj = (long)(d.IM - 2) * (d.JM - 1) * (d.KM - 2);
  const long nfk = (long)(d.IM - 2) * (d.JM - 2) * (d.KM - 1);
  *first = kind == 0 ? 0 : (kind == 1 ? nfi : nfi + nfj);
  *count = kind == 0 ? nfi : (kind == 1 ? nfj : nfk);
}

// A face of a's stage input: its index, low node and kind, from entry w of the
// list or (with all set) face w of the block.
struct FaceRef {
  long e, oa;
  int kind;
};
__device__ __forceinline__ FaceRef face_ref(const Dims& d, bool all, long w, const int2* list) {
  if (all) {  // decoded by 32-bit divisions (fewer than 2^31 faces), i fastest
    long first = 0, count;
    int kind = 2;
    for (; kind >= 0; --kind) {
      kind_range(d, kind, &first, &count);
      if (w >= first) break;
    }
    const unsigned ni = (unsigned)(kind == 0 ? d.IM - 1 : d.IM - 2), nj = (unsigned)(kind == 1 ? d.JM - 1 : d.JM - 2);
    const unsigned u = (unsigned)(w - first), r = u / ni, k = r / nj;
    return FaceRef{w, node_off(d, (int)(u - r * ni) + (kind != 0), (int)(r - k * nj) + (kind != 1), (int)k + (kind != 2)),
                   kind};
  }
  const int2 le = __ldg(list + w);
  return FaceRef{le.x, (long)((unsigned)le.y & 0x3fffffffu), (int)((unsigned)le.y >> 30)};
}

// The WENO5 fluxes of the two faces w0 and w1 (the same kind) into a.wflux.
// Each thread stages its pair's stencil values in its own column of shared
// memory (my, stride WT), so the packed flux reads them there, pairs in one
// load, instead of keeping them in registers.
__device__ __forceinline__ void weno_pair(const StageArgs& a, bool all, long w0, long w1, const int2* list, float2* my) {
  const Dims& d = a.d;
  const FaceRef r0 = face_ref(d, all, w0, list), r1 = face_ref(d, all, w1, list);
  // along the face normal: the stride s; area vector components 3*kind ..
  const long s = r0.kind == 0 ? 1 : r0.kind == 1 ? d.PX : d.PL;
  {
    const float *p0 = a.src32 + r0.oa - 2 * s, *p1 = a.src32 + r1.oa - 2 * s;
#pragma unroll
    for (int q = 0; q < NEQ; ++q)
#pragma unroll
      for (int p = 0; p < 6; ++p)
        my[(q * 6 + p) * WT] = make_float2(__ldg(p0 + q * d.VOL + p * s), __ldg(p1 + q * d.VOL + p * s));
  }
  F2 n[3];
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    const float* ar = a.area32[0] + (3 * r0.kind + m) * d.VOL;
    n[m] = mk(0.5f * (__ldg(ar + r0.oa) + __ldg(ar + r0.oa + s)), 0.5f * (__ldg(ar + r1.oa) + __ldg(ar + r1.oa + s)));
  }
  auto ld = [&](int p, int q) -> F2 {
    const float2 v = my[(q * 6 + p) * WT];
    return mk(v.x, v.y);
  };
  const FluxConsts<float> C{(float)a.gamma, (float)a.gam1, (float)a.gam1_inv};
  F2 f[5];
  face_flux<F2>(ld, n[0], n[1], n[2], C, f);
  float x[5], y[5];
#pragma unroll
  for (int m = 0; m < NEQ; ++m) halves(f[m], x[m], y[m]);
  auto put = [&](long e, const float* v) {
    float* out = a.wflux + 8 * e;
    *reinterpret_cast<float4*>(out) = make_float4(v[0], v[1], v[2], v[3]);
    out[4] = v[4];
  };
  put(r0.e, x);
  put(r1.e, y);
}

// Two listed faces per thread (faces while force_weno is set), WT apart in the
// list so that neighbouring threads read neighbouring faces.  The CTAs are
// shared out among the three kinds' lists in proportion to their lengths (at
// least one for a kind with faces), and each kind's CTAs walk its list
// grid-stride, so the three kinds advance through the grid's planes side by
// side and the stencils they share stay in L2.  A list of odd length ends with
// its last face evaluated twice by one thread.
// Bound by the stencil loads (24% of issue slots idle on them) and the FP32
// pipe.  Built for 3 CTAs of 128 threads per SM (168 registers).  One launch of
// a 256x256x128 hybrid step: 171 us with one face per thread from the FP64
// state (256 threads, 80 registers), 149 us in pairs from its FP32 copy (152
// with a reciprocal per indicator, face_flux.cuh).
__global__ void __launch_bounds__(WT, 3) weno_faces_kernel(const __grid_constant__ StageArgs a, int mode,
                                                           const int2* list) {
  __shared__ float2 stn[NEQ * 6][WT];
  const StepState* st = a.st;
  if (mode != 0 && st->done) return;
  const bool all = st->force_weno != 0;
  long first[3], len[3];
  for (int k = 0; k < 3; ++k) {
    long cnt;
    kind_range(a.d, k, &first[k], &cnt);
    len[k] = all ? cnt : (long)st->weno_listed[k];
  }
  const long tot = len[0] + len[1] + len[2];
  if (tot == 0) return;
  const int G = gridDim.x;
  int b1 = (int)((len[0] * G + tot - 1) / tot), b2 = (int)(((len[0] + len[1]) * G + tot - 1) / tot);
  b1 = min(max(b1, len[0] > 0 ? 1 : 0), G - (len[1] > 0 ? 1 : 0) - (len[2] > 0 ? 1 : 0));
  b2 = min(max(b2, b1 + (len[1] > 0 ? 1 : 0)), G - (len[2] > 0 ? 1 : 0));
  const int c = blockIdx.x;
  const int k = c < b1 ? 0 : (c < b2 ? 1 : 2);
  const int base = k == 0 ? 0 : (k == 1 ? b1 : b2);
  const int g = k == 0 ? b1 : (k == 1 ? b2 - b1 : G - b2);
  for (long w = (long)(c - base) * 2 * WT + threadIdx.x; w < len[k]; w += (long)g * 2 * WT)
    weno_pair(a, all, first[k] + w, first[k] + min(w + WT, len[k] - 1), list, &stn[0][threadIdx.x]);
}

int g_weno_grid = 0;  // persistent grid of the evaluation kernel: resident CTAs of the device

}  // namespace

cudaError_t weno_prepare() {
  if (g_weno_grid) return cudaSuccess;
  int per_sm = 0, dev = 0, nsm = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, weno_faces_kernel, WT, 0);
  if (e == cudaSuccess) e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  g_weno_grid = nsm * (per_sm > 0 ? per_sm : 1);
  return cudaSuccess;
}

cudaError_t launch_weno_faces(const StageArgs& a, int mode, long nfaces, const int2* list, cudaStream_t s) {
  cudaError_t e = weno_prepare();
  if (e != cudaSuccess || nfaces <= 0) return e;
  weno_faces_kernel<<<g_weno_grid, WT, 0, s>>>(a, mode, list);
  return cudaGetLastError();
}

}  // namespace cbns
