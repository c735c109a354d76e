// sensor.cu - training side of the learned shock sensor: face sampling with
// features and WENO-weight labels from a solver state, the network's loss and
// gradient over a batch (forward and backward by hand), the Adam update, and
// an FP32 forward pass.  See sensor.cuh for the features, label and layout.
#include "face_flux.cuh"
#include "sensor.cuh"
#include "sensor_kernels.cuh"

namespace cbns {

namespace {

// ---------------------------------------------------------------- sampling
__global__ void sample_faces_kernel(const SampleArgs a) {
  const Dims& d = a.d;
  const long ni = (long)(d.IM - 1) * (d.JM - 2) * (d.KM - 2);
  const long nj = (long)(d.IM - 2) * (d.JM - 1) * (d.KM - 2);
  const long nk = (long)(d.IM - 2) * (d.JM - 2) * (d.KM - 1);
  const long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (e >= ni + nj + nk || (e % a.stride) != a.offset) return;
  int dir, i, j, k;
  if (e < ni) {  // face between (i, j+1, k+1) and (i+1, j+1, k+1)
    dir = 0;
    i = (int)(e % (d.IM - 1));
    j = 1 + (int)((e / (d.IM - 1)) % (d.JM - 2));
    k = 1 + (int)(e / ((long)(d.IM - 1) * (d.JM - 2)));
  } else if (e < ni + nj) {
    const long r = e - ni;
    dir = 1;
    i = 1 + (int)(r % (d.IM - 2));
    j = (int)((r / (d.IM - 2)) % (d.JM - 1));
    k = 1 + (int)(r / ((long)(d.IM - 2) * (d.JM - 1)));
  } else {
    const long r = e - ni - nj;
    dir = 2;
    i = 1 + (int)(r % (d.IM - 2));
    j = 1 + (int)((r / (d.IM - 2)) % (d.JM - 2));
    k = (int)(r / ((long)(d.IM - 2) * (d.JM - 2)));
  }
  const long sd = dir == 0 ? 1 : (dir == 1 ? d.PX : d.PL);
  const long oa = node_off(d, i, j, k), ob = oa + sd;
  const double* q = a.q;
  const long V = d.VOL;
  auto ld = [&](int p, int n) -> float { return (float)q[n * V + oa + (p - 2) * sd]; };
  // the same FP32 arithmetic as the per-step sensor sweep, so that inference
  // sees exactly the features the network was trained on
  float A[3], B[3];
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    A[m] = (float)node_area(a.met, 3 * dir + m, oa);
    B[m] = (float)node_area(a.met, 3 * dir + m, ob);
  }
  float ux, uy, uz;
  face_unit_normal(A, B, ux, uy, uz);
  float f[SN_IN];
  face_features(ld, ux, uy, uz, a.gamma, a.gam1, f);
  const float dev = face_weno_deviation(ld, 0.5f * (A[0] + B[0]), 0.5f * (A[1] + B[1]), 0.5f * (A[2] + B[2]),
                                        a.gamma, a.gam1);
  const unsigned slot = atomicAdd(a.count, 1u);
  if (slot >= a.capacity) return;
#pragma unroll
  for (int m = 0; m < SN_IN; ++m) a.feat[(long)slot * SN_IN + m] = f[m];
  a.label[slot] = dev > SN_DEV_THRESHOLD ? 1 : 0;
  if (a.dev) a.dev[slot] = dev;
  if (a.index) a.index[slot] = (unsigned)e;
}

// ---------------------------------------------------------------- loss and gradient
constexpr int TILE = 64, GT = 256;
constexpr int HP = SN_H + 4, XP = 20;  // row pitches: 16-byte rows, four rows apart in different banks

static_assert(TILE * HP > SP_N && TILE * XP >= SN_H * 16, "the gradients fit the tile's buffers");

struct GradSmem {
  alignas(16) float x[TILE][XP];
  alignas(16) float h1[TILE][HP], h2[TILE][HP], g2[TILE][HP], g1[TILE][HP];
  alignas(16) float W2[SN_H][HP];
  float dz[TILE];
  float w3[SN_H];
};

// Binary cross-entropy with positive-class weight, averaged over n samples:
// loss = -(1/n) sum w_i [y_i log p_i + (1 - y_i) log(1 - p_i)], p = sigmoid(z).
// Each CTA takes tiles of 64 samples: forward into shared memory, backward by
// the chain rule, per-thread partial sums of the weight gradients in registers,
// one atomic add per parameter per CTA at the end.  Bound by the latency of a
// tile's chain of phases: a training batch (16,384 samples) is one tile for each
// of 256 CTAs, so the tile is small, rows are read as float4 (broadcast), the
// weight gradients take 2 x 2 outputs per thread (two 8-byte reads for four
// products) and the last layer shares its sums among four threads a row.
// 16,384 samples: 20.3 -> 12.8 us (128 tiles of 128 samples before; weights
// loaded across their rows), 1.5 M samples 1050 -> 686 us; summing over clusters
// of 4 or 8 CTAs first was slower (15.0 and 17.7 us, 1213 us).
__global__ void __launch_bounds__(GT) mlp_grad_kernel(const float* __restrict__ P, const float* __restrict__ X,
                                                      const unsigned char* __restrict__ Y, unsigned n, float pos_w,
                                                      float inv_n, float* G, float* loss) {
  extern __shared__ __align__(16) unsigned char raw[];
  GradSmem& s = *reinterpret_cast<GradSmem*>(raw);
  const int t = threadIdx.x;
  const int c = t & 31, rb = t >> 5;  // column and first row of this thread's outputs
  // the weights through shared memory (a thread's rows of them straight from
  // memory are 47 loads of 32 sectors each, 6 us a CTA)
  for (int e = t; e < SN_H * SN_H; e += GT) s.W2[e / SN_H][e % SN_H] = P[SP_W2 + e];
  for (int e = t; e < SN_H * SN_IN; e += GT) s.x[e / SN_IN][e % SN_IN] = P[SP_W1 + e];
  if (t < SN_H) {
    s.w3[t] = P[SP_W3 + t];
    s.x[t][SN_IN] = 0.f;
  }
  __syncthreads();
  float w1[SN_IN + 1], w2[SN_H];
#pragma unroll
  for (int k = 0; k < SN_IN + 1; ++k) w1[k] = s.x[c][k];
#pragma unroll
  for (int k = 0; k < SN_H; ++k) w2[k] = s.W2[c][k];
  const float b1 = P[SP_B1 + c], b2 = P[SP_B2 + c], b3 = P[SP_B3];
  // owned gradient entries: a 2 x 2 block of W2 (rows 2i.., columns 2j..), of W1
  // (columns below 15; threads below 128), and one entry of the vectors
  const int bi = 2 * (t >> 4), bj = 2 * (t & 15);
  const int ai = 2 * ((t & 127) >> 3), aj = 2 * (t & 7);
  float gW2[2][2] = {{0.f, 0.f}, {0.f, 0.f}}, gW1[2][2] = {{0.f, 0.f}, {0.f, 0.f}}, gvec = 0.f, lsum = 0.f;
  __syncthreads();
  auto dot4 = [](const float4 a, const float* w, float h) {
    h += a.x * w[0];
    h += a.y * w[1];
    h += a.z * w[2];
    return h + a.w * w[3];
  };
  const unsigned ntiles = (n + TILE - 1) / TILE;
  for (unsigned tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const unsigned base = tile * TILE;
    for (int e = t; e < TILE * SN_IN; e += GT) {  // the tile's features are contiguous
      const int r = e / SN_IN, k = e % SN_IN;
      s.x[r][k] = base + r < n ? X[(size_t)base * SN_IN + e] : 0.f;
    }
    if (t < TILE) s.x[t][SN_IN] = 0.f;
    __syncthreads();
#pragma unroll 4
    for (int r = rb; r < TILE; r += GT / 32) {
      const float4* xr = reinterpret_cast<const float4*>(s.x[r]);
      float h = b1;
#pragma unroll
      for (int k = 0; k < 4; ++k) h = dot4(xr[k], w1 + 4 * k, h);
      s.h1[r][c] = fmaxf(h, 0.f);
    }
    __syncthreads();
#pragma unroll 4
    for (int r = rb; r < TILE; r += GT / 32) {
      const float4* hr = reinterpret_cast<const float4*>(s.h1[r]);
      float h = b2;
#pragma unroll
      for (int k = 0; k < SN_H / 4; ++k) h = dot4(hr[k], w2 + 4 * k, h);
      s.h2[r][c] = fmaxf(h, 0.f);
    }
    __syncthreads();
    {  // the logit, loss and its derivative: row t / 4, a quarter of the sum each
      const int r = t >> 2, q = t & 3;
      const unsigned sidx = base + r;
      float z = 0.f;
#pragma unroll
      for (int k = 0; k < SN_H / 4; ++k) z += s.h2[r][4 * k + q] * s.w3[4 * k + q];
      z += __shfl_xor_sync(0xffffffffu, z, 1);
      z += __shfl_xor_sync(0xffffffffu, z, 2);
      z += b3;
      if (q == 0) {
        float dz = 0.f;
        if (sidx < n) {
          const float y = Y[sidx] ? 1.f : 0.f;
          const float w = Y[sidx] ? pos_w : 1.f;
          const float p = 1.f / (1.f + __expf(-z));
          // log(sigmoid(z)) and log(1 - sigmoid(z)) in a form that does not overflow
          const float lp = -log1pf(__expf(-fabsf(z))) + fminf(z, 0.f);
          const float lq = lp - z;
          lsum += -w * (y * lp + (1.f - y) * lq) * inv_n;
          dz = w * (p - y) * inv_n;
        }
        s.dz[r] = dz;
      }
    }
    __syncthreads();
    for (int r = rb; r < TILE; r += GT / 32) s.g2[r][c] = s.h2[r][c] > 0.f ? s.dz[r] * s.w3[c] : 0.f;
    __syncthreads();
    // dW2[cc][k] = sum_r g2[r][cc] h1[r][k]
    {
      float a00 = 0.f, a01 = 0.f, a10 = 0.f, a11 = 0.f;
#pragma unroll 8
      for (int r = 0; r < TILE; ++r) {
        const float2 g = *reinterpret_cast<const float2*>(&s.g2[r][bi]), h = *reinterpret_cast<const float2*>(&s.h1[r][bj]);
        a00 += g.x * h.x;
        a01 += g.x * h.y;
        a10 += g.y * h.x;
        a11 += g.y * h.y;
      }
      gW2[0][0] += a00;
      gW2[0][1] += a01;
      gW2[1][0] += a10;
      gW2[1][1] += a11;
    }
    // per-column vectors: db2 (32..63), dw3 (64..95), db3 (96); db1 after g1
    if (t >= 32 && t < 64) {
      float acc = 0.f;
#pragma unroll 8
      for (int r = 0; r < TILE; ++r) acc += s.g2[r][t - 32];
      gvec += acc;
    } else if (t >= 64 && t < 96) {
      float acc = 0.f;
#pragma unroll 8
      for (int r = 0; r < TILE; ++r) acc += s.dz[r] * s.h2[r][t - 64];
      gvec += acc;
    } else if (t == 96) {
      float acc = 0.f;
#pragma unroll 8
      for (int r = 0; r < TILE; ++r) acc += s.dz[r];
      gvec += acc;
    }
    // g1[r][k] = (sum_c g2[r][c] W2[c][k]) * relu'(h1)
    {
      float w2c[SN_H];
#pragma unroll
      for (int cc = 0; cc < SN_H; ++cc) w2c[cc] = s.W2[cc][c];
#pragma unroll 4
      for (int r = rb; r < TILE; r += GT / 32) {
        const float4* gr = reinterpret_cast<const float4*>(s.g2[r]);
        float acc = 0.f;
#pragma unroll
        for (int k = 0; k < SN_H / 4; ++k) acc = dot4(gr[k], w2c + 4 * k, acc);
        s.g1[r][c] = s.h1[r][c] > 0.f ? acc : 0.f;
      }
    }
    __syncthreads();
    // dW1, by two halves of the rows (threads 0..127 and 128..255)
    {
      const int r0 = t < 128 ? 0 : TILE / 2;
      float a00 = 0.f, a01 = 0.f, a10 = 0.f, a11 = 0.f;
#pragma unroll 8
      for (int r = r0; r < r0 + TILE / 2; ++r) {
        const float2 g = *reinterpret_cast<const float2*>(&s.g1[r][ai]), x = *reinterpret_cast<const float2*>(&s.x[r][aj]);
        a00 += g.x * x.x;
        a01 += g.x * x.y;
        a10 += g.y * x.x;
        a11 += g.y * x.y;
      }
      gW1[0][0] += a00;
      gW1[0][1] += a01;
      gW1[1][0] += a10;
      gW1[1][1] += a11;
    }
    if (t < 32) {
      float acc = 0.f;
#pragma unroll 8
      for (int r = 0; r < TILE; ++r) acc += s.g1[r][t];
      gvec += acc;
    }
    __syncthreads();
  }
  // the CTA's gradients (and the loss at index SP_N) through shared memory, so
  // that neighbouring threads add to neighbouring parameters
  float* own = &s.h1[0][0];  // TILE x HP >= SP_N + 1 floats; the loop's last barrier freed it
#pragma unroll
  for (int p = 0; p < 2; ++p)
#pragma unroll
    for (int q = 0; q < 2; ++q) own[SP_W2 + (bi + p) * SN_H + bj + q] = gW2[p][q];
  if (t >= 128) {  // the second half of the rows' share of W1
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
      for (int q = 0; q < 2; ++q) s.x[0][(ai + p) * 16 + aj + q] = gW1[p][q];
  }
  if (t < 32) own[SP_B1 + t] = gvec;
  else if (t < 64) own[SP_B2 + t - 32] = gvec;
  else if (t < 96) own[SP_W3 + t - 64] = gvec;
  else if (t == 96) own[SP_B3] = gvec;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
  if ((t & 31) == 0) s.dz[t >> 5] = lsum;
  __syncthreads();
  if (t < 128) {
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
      for (int q = 0; q < 2; ++q)
        if (aj + q < SN_IN) own[SP_W1 + (ai + p) * SN_IN + aj + q] = gW1[p][q] + s.x[0][(ai + p) * 16 + aj + q];
  }
  if (t == 0) {
    float l = 0.f;
    for (int w = 0; w < GT / 32; ++w) l += s.dz[w];
    own[SP_N] = l;
  }
  __syncthreads();
  for (int e = t; e <= SP_N; e += GT) atomicAdd(e < SP_N ? G + e : loss, own[e]);
}

__global__ void zero_grad(float* G, float* loss) {
  const int e = blockIdx.x * 256 + threadIdx.x;
  if (e < SP_N) G[e] = 0.f;
  else if (e == SP_N) *loss = 0.f;
}

// ---------------------------------------------------------------- widening
// Both passes take one 32-face word per thread, DT threads per CTA.  Three
// passes of a load per face and window place on bytes, and one that listed the
// faces from the bytes, took 207 + 55 us per network step on a 256x256x128
// grid.  On bits 32 faces share every load and OR, and the words that pass 1
// has in registers give the list: 18 + 37 us, the rest the 25 MB of bytes and
// their 32 warp-wide stores per warp of words.
constexpr int DT = 256;

// the kind and the place (word of the line, line indices) of word w
__device__ __forceinline__ BitRows bit_place(const Dims& d, long w, int& kind, int& x, int& j, int& k) {
  BitRows b = bit_rows(d, 2);
  kind = 2;
  while (w < b.word) b = bit_rows(d, --kind);
  const unsigned r = (unsigned)(w - b.word), line = r / (unsigned)b.W;
  x = (int)(r - line * (unsigned)b.W);
  k = (int)(line / (unsigned)b.n1);
  j = (int)(line - (unsigned)k * (unsigned)b.n1);
  return b;
}

// pass 0 or 1 for the CTA bx of one block's grid
template <int PASS>
__device__ __forceinline__ void dilate_body(const DilateArgs& a, unsigned bx) {
  if (a.check_done && a.st->done) return;
  const bool lead = bx == 0 && threadIdx.x == 0;
  if (a.hold || !sensor_step(a.st, a.every)) {
    // decisions of an earlier step: only the statistics, that step's count
    if (PASS == 1 && lead) atomicAdd(&a.st->weno_faces, a.st->weno_last);
    return;
  }
  if (PASS == 0 && lead) {  // pass 1 counts and lists anew
    a.st->weno_last = 0;
    for (int m = 0; m < 3; ++m) a.st->weno_listed[m] = 0;
  }
  const Dims& d = a.d;
  const long words = bit_words(d), w = (long)bx * DT + threadIdx.x;
  int kind = 0, x = 0, j = 0, k = 0;
  BitRows b{};
  unsigned v = 0;
  if (PASS == 0) {
    if (w >= words) return;
    b = bit_place(d, w, kind, x, j, k);
    // OR of the lines j - wj .. j + wj, then of the faces x - wi .. x + wi of it
    const int wi = kind == 0 ? a.along : a.across, wj = kind == 1 ? a.along : a.across;
    unsigned prev = 0, cur = 0, next = 0;
    const unsigned* p = a.in + b.word + (long)k * b.n1 * b.W + x;
    for (int jj = max(0, j - wj); jj <= min(b.n1 - 1, j + wj); ++jj) {
      const unsigned* q = p + (long)jj * b.W;
      cur |= __ldg(q);
      if (x > 0) prev |= __ldg(q - 1);
      if (x + 1 < b.W) next |= __ldg(q + 1);
    }
    v = cur;
    for (int s = 1; s <= wi; ++s) v |= __funnelshift_l(prev, cur, s) | __funnelshift_r(cur, next, s);
    const int n = b.n0 - 32 * x;  // faces of the line's last word
    if (n < 32) v &= (1u << n) - 1u;
    a.mid[w] = v;
  } else {
    __shared__ int wcnt[3][DT / 32], base[3];
    int e = 0, n = 0;
    unsigned oa = 0;
    if (w < words) {
      b = bit_place(d, w, kind, x, j, k);
      const int wk = kind == 2 ? a.along : a.across;
      const long plane = (long)b.n1 * b.W;
      const unsigned* p = a.mid + w;
      for (int kk = max(0, k - wk); kk <= min(b.n2 - 1, k + wk); ++kk) v |= __ldg(p + (kk - k) * plane);
      e = (int)(b.face + ((long)k * b.n1 + j) * b.n0 + 32 * x);
      n = min(32, b.n0 - 32 * x);
      oa = (unsigned)node_off(d, 32 * x + (kind != 0), j + (kind != 1), k + (kind != 2));  // low node of the word's first face
    }
    // where each word's faces go in its kind's list: a scan over the warp, then
    // over the CTA's warps, and one atomic per kind that the CTA meets
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int pos = 0;
    for (int m = 0; m < 3; ++m) {
      const int c = kind == m ? __popc(v) : 0;
      int incl = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      if (kind == m) pos = incl - c;
      if (lane == 31) wcnt[m][warp] = incl;
    }
    __syncthreads();
    if (threadIdx.x < 3) {
      const int m = threadIdx.x;
      int tot = 0;
      for (int q = 0; q < DT / 32; ++q) {
        const int c = wcnt[m][q];
        wcnt[m][q] = tot;
        tot += c;
      }
      if (tot) {
        base[m] = (int)bit_rows(d, m).face + (int)atomicAdd(&a.st->weno_listed[m], (unsigned)tot);
        atomicAdd(&a.st->weno_faces, (unsigned long long)tot);
        atomicAdd(&a.st->weno_last, (unsigned long long)tot);
      }
    }
    __syncthreads();
    pos += base[kind] + wcnt[kind][warp];
    // each lane's word as 32 bytes and its list entries, the warp on one word
    // at a time
    for (int s = 0; s < 32; ++s) {
      const int ns = __shfl_sync(0xffffffffu, n, s), es = __shfl_sync(0xffffffffu, e, s);
      const unsigned vs = __shfl_sync(0xffffffffu, v, s);
      const bool on = (vs >> lane) & 1u;
      if (lane < ns) a.out[es + lane] = on;
      if (vs) {
        const int ps = __shfl_sync(0xffffffffu, pos, s), ks = __shfl_sync(0xffffffffu, kind, s);
        const unsigned os = __shfl_sync(0xffffffffu, oa, s);
        if (on) a.list[ps + __popc(vs & ((1u << lane) - 1u))] = list_entry(es + lane, ks, os + lane);
      }
    }
  }
}

template <int PASS>
__global__ void __launch_bounds__(DT) sensor_dilate_kernel(const DilateArgs a) {
  dilate_body<PASS>(a, blockIdx.x);
}

// Many blocks in one launch: block b owns CTAs cta[b] .. cta[b+1]-1, args[b]
// are its DilateArgs.
template <int PASS>
__global__ void __launch_bounds__(DT) sensor_dilate_batched(const DilateArgs* args, const int* cta, int nblocks) {
  const int b = block_of_cta(cta, nblocks, (int)blockIdx.x);
  dilate_body<PASS>(args[b], blockIdx.x - (unsigned)__ldg(cta + b));
}

// ---------------------------------------------------------------- audit
__device__ __forceinline__ void audit_body(const AuditArgs& a, unsigned bx) {
  if (a.check_done && a.st->done) return;
  const Dims& d = a.d;
  const long nf = total_faces(d);
  // runs of 128 consecutive faces (coalesced loads): run r is audited when
  // r % stride == steps % stride
  const unsigned off = a.st->steps % a.stride;
  const long e = ((long)bx * a.stride + off) * 128 + threadIdx.x;
  float err = 0.f;
  bool audited = false;
  int dir, i, j, k;
  if (e < nf && a.mask[e] == 0 && decode_face(d, e, dir, i, j, k)) {
    const long sd = dir == 0 ? 1 : (dir == 1 ? d.PX : d.PL);
    const long oa = node_off(d, i, j, k), ob = oa + sd;
    auto ld = [&](int p, int n) -> float { return __ldg(a.q + n * d.VOL + oa + (p - 2) * sd); };
    auto normal = [&](int m) { return (float)(0.5 * (node_area(a.met, m, oa) + node_area(a.met, m, ob))); };
    const float nx = normal(3 * dir), ny = normal(3 * dir + 1), nz = normal(3 * dir + 2);
    const FluxConsts<float> C{a.gamma, a.gam1, a.gam1_inv};
    float fw[5], fl[5];
    face_flux<float>(ld, nx, ny, nz, C, fw);
    face_flux_linear<float>(ld, nx, ny, nz, C, fl);
    float num = 0.f, den = 0.f;
#pragma unroll
    for (int n = 0; n < 5; ++n) {
      num = fmaxf(num, fabsf(fw[n] - fl[n]));
      den = fmaxf(den, fabsf(fw[n]));
    }
    err = num / (den + 1.0e-20f);
    if (!(err == err)) err = 3.0e38f;
    audited = true;
  }
  // one set of atomics per CTA, the maximum's only where it grows
  __shared__ float wmax[4];
  float m = err;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = m;
  const int n_aud = __syncthreads_count(audited);
  if (threadIdx.x == 0 && n_aud) {
    m = fmaxf(fmaxf(wmax[0], wmax[1]), fmaxf(wmax[2], wmax[3]));
    atomicAdd(&a.st->audit_faces, (unsigned long long)n_aud);
    if (m > *(volatile float*)&a.st->audit_max)
      atomicMax(reinterpret_cast<int*>(&a.st->audit_max), __float_as_int(m));  // m >= 0: int order = float order
    if (m > a.bound && atomicExch(&a.st->force_weno, 1) == 0) atomicAdd(&a.st->audit_fail_steps, 1u);
  }
}

__global__ void __launch_bounds__(128) sensor_audit_kernel(const AuditArgs a) { audit_body(a, blockIdx.x); }

__global__ void __launch_bounds__(128) sensor_audit_batched(const AuditArgs* args, const int* cta, int nblocks) {
  const int b = block_of_cta(cta, nblocks, (int)blockIdx.x);
  audit_body(args[b], blockIdx.x - (unsigned)__ldg(cta + b));
}

__global__ void adam_kernel(float* P, const float* G, float* M, float* V, float lr, float c1, float c2) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= SP_N) return;
  const float g = G[e];
  const float m = 0.9f * M[e] + 0.1f * g;
  const float v = 0.999f * V[e] + 0.001f * g * g;
  M[e] = m;
  V[e] = v;
  P[e] -= lr * (m * c1) / (sqrtf(v * c2) + 1.0e-8f);
}

__global__ void mlp_predict_kernel(const float* __restrict__ P, const float* __restrict__ X, unsigned n,
                                   float* __restrict__ out) {
  __shared__ float sp[SP_N];
  for (int e = threadIdx.x; e < SP_N; e += blockDim.x) sp[e] = P[e];
  __syncthreads();
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float x[SN_IN];
#pragma unroll
  for (int k = 0; k < SN_IN; ++k) x[k] = X[(size_t)i * SN_IN + k];
  out[i] = 1.f / (1.f + __expf(-mlp_forward(sp, x)));
}

}  // namespace

cudaError_t launch_sample_faces(const SampleArgs& a, cudaStream_t s) {
  const Dims& d = a.d;
  const long n = (long)(d.IM - 1) * (d.JM - 2) * (d.KM - 2) + (long)(d.IM - 2) * (d.JM - 1) * (d.KM - 2) +
                 (long)(d.IM - 2) * (d.JM - 2) * (d.KM - 1);
  sample_faces_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(a);
  return cudaGetLastError();
}

int sensor_audit_ctas(const AuditArgs& a) {
  const long nf = (long)(a.d.IM - 1) * (a.d.JM - 2) * (a.d.KM - 2) + (long)(a.d.IM - 2) * (a.d.JM - 1) * (a.d.KM - 2) +
                  (long)(a.d.IM - 2) * (a.d.JM - 2) * (a.d.KM - 1);
  const long runs = (nf + 127) / 128;
  return (int)((runs + a.stride - 1) / a.stride);
}

cudaError_t launch_sensor_audit(const AuditArgs& a, cudaStream_t s) {
  sensor_audit_kernel<<<(unsigned)sensor_audit_ctas(a), 128, 0, s>>>(a);
  return cudaGetLastError();
}

int sensor_dilate_ctas(const Dims& d) { return (int)((bit_words(d) + DT - 1) / DT); }

cudaError_t launch_sensor_dilate(const DilateArgs& a, int pass, cudaStream_t s) {
  const int ctas = sensor_dilate_ctas(a.d);
  if (pass == 0) sensor_dilate_kernel<0><<<ctas, DT, 0, s>>>(a);
  else sensor_dilate_kernel<1><<<ctas, DT, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_sensor_audit_batched(const AuditArgs* args, const int* cta, int nblocks, int total,
                                        cudaStream_t s) {
  if (total <= 0) return cudaSuccess;
  sensor_audit_batched<<<total, 128, 0, s>>>(args, cta, nblocks);
  return cudaGetLastError();
}

cudaError_t launch_sensor_dilate_batched(const DilateArgs* args, const int* cta, int nblocks, int total, int pass,
                                         cudaStream_t s) {
  if (total <= 0) return cudaSuccess;
  if (pass == 0) sensor_dilate_batched<0><<<total, DT, 0, s>>>(args, cta, nblocks);
  else sensor_dilate_batched<1><<<total, DT, 0, s>>>(args, cta, nblocks);
  return cudaGetLastError();
}

cudaError_t launch_mlp_grad(const float* P, const float* X, const unsigned char* Y, unsigned n, float pos_w, float* G,
                            float* loss, cudaStream_t s) {
  zero_grad<<<(SP_N + 256) / 256, 256, 0, s>>>(G, loss);  // one launch for two memsets
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  if (n == 0) return cudaSuccess;
  static bool attr = false;
  if (!attr) {
    e = cudaFuncSetAttribute(mlp_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(GradSmem));
    if (e != cudaSuccess) return e;
    attr = true;
  }
  const unsigned ntiles = (n + TILE - 1) / TILE;
  const unsigned grid = ntiles < 296u ? ntiles : 296u;
  mlp_grad_kernel<<<grid, GT, sizeof(GradSmem), s>>>(P, X, Y, n, pos_w, 1.0f / (float)n, G, loss);
  return cudaGetLastError();
}

cudaError_t launch_adam(float* P, const float* G, float* M, float* V, unsigned step, float lr, cudaStream_t s) {
  const float c1 = 1.0f / (1.0f - powf(0.9f, (float)step));
  const float c2 = 1.0f / (1.0f - powf(0.999f, (float)step));
  adam_kernel<<<(SP_N + 255) / 256, 256, 0, s>>>(P, G, M, V, lr, c1, c2);
  return cudaGetLastError();
}

cudaError_t launch_mlp_predict(const float* P, const float* X, unsigned n, float* out, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  mlp_predict_kernel<<<(n + 255) / 256, 256, 0, s>>>(P, X, n, out);
  return cudaGetLastError();
}

}  // namespace cbns
