// stage.cuh - launch interface of the fused RK3 stage kernel (stage.cu).
#pragma once

#include <cuda.h>

#include "cbns_common.cuh"
#include "kchunk.h"
#include "tma.cuh"

namespace cbns {

// TMA tensor maps of the stage kernels (tma.cuh), 4-D: x, rows, planes,
// fields.  q_a: the ring column box (16 x 15 x 1 x 5) of the stage input, q_b
// its plane-with-halo box (24 x 21 x 1 x 5), xi / eta the face-node area
// vectors (24 x 15 x 1 x 3 and 16 x 17 x 1 x 3), zeta (16 x 15 x 1 x 3): FP64 in
// the FP64 kernel (the 10 area components), FP32 copies in the FP32 kernels
// (the 9 area32 components).  The FP64 update operands' boxes (16 x 15 x 1 x 5,
// iJ x 1), prefetched into L2: q0, qp, iJ, and in the FP32 kernels of viscous
// runs dfv (FP32 elements, x 4).
struct StageMaps {
  CUtensorMap q_a, q_b, xi, eta, zeta, q0, qp, iJ, dfv;
};
constexpr int kStageMaps = sizeof(StageMaps) / sizeof(CUtensorMap);

struct StageCore {
  Dims d;
  double gamma, gam1, gam1_inv, gM2;
  const double* src;   // stage input (stencil source), 5 fields
  const double* q0;    // the reference's Q at the node (RK base)
  const double* qp;    // the reference's Q_p at the node (stages 2, 3)
  double* out;         // stage output (5 fields), or the dense RHS array in mode 0
  float* out32;        // FP32 kernels: the FP32 copy of the stage output
  const float* src32;  // FP32 kernels: the FP32 copy of the stage input
  const double* area[10];  // J*grad(xi|eta|zeta) per node, then 1/J
  const double* dfv[4];    // viscous: the divergence of the node fluxes (visc.cu; FP32 elements in the FP32 kernels)
  double* prim[6];     // viscous: rho,u,v,w,p,T of the new interior state
  StepState* st;       // dt, done flag, spectral-radius max
  const unsigned char* mask;  // hybrid: per-face sensor decision (null: plain flux everywhere)
  float* wflux;        // hybrid: WENO5 flux of each WENO5 face (8 floats per face, 5 used)
  const float* area32[9];  // FP32 kernels: J*grad(xi), J*grad(eta), J*grad(zeta) per node in FP32
  int q0_is_src, qp_is_src;  // RK operands that equal the stage input (read from the ring)
  int ntile_i, ntile_j, kchunk;
  int lean;            // viscous, stages 1 and 2 of a run: rho and p of the primitives are not read before stage 3
  int sigma;           // accumulate the interior spectral-radius max (inviscid stage 3)
};
struct StageArgs : StageCore {
  StageMaps tm;
};

// A batch item's StageCore from the device table into shared memory (its tensor
// maps are read where they lie); nt threads.
__device__ __forceinline__ void copy_core(StageCore* to, const StageCore* from, int nt) {
  const int* src = reinterpret_cast<const int*>(from);
  int* dst = reinterpret_cast<int*>(to);
  for (int e = threadIdx.x; e < (int)(sizeof(StageCore) / sizeof(int)); e += nt) dst[e] = __ldg(src + e);
}

// The tensor maps of batch item `blk`, once per CTA and block (thread 0, which
// alone uses them; `have`: the block of its last item, -1 at first).
__device__ __forceinline__ void batch_maps(const StageArgs* args, int blk, int& have) {
  if (threadIdx.x != 0 || blk == have) return;
  have = blk;
  tma::acquire_maps(&args[blk].tm.q_a, kStageMaps);
}

// Many blocks in one launch (a persistent work queue): args[b] are the
// StageArgs of block b, its work items (tile, k chunk) are numbered
// start[b] .. start[b+1]-1 of total, and *counter (zeroed before the launch)
// hands them out.
struct BatchStage {
  const StageArgs* args;  // device, nblocks entries
  const int* start;       // device, nblocks + 1 entries
  int nblocks, total;
  unsigned* counter;      // device
};

// mode 0: dense RHS output; 1..3: RK stage.  fp32: split-precision flux arithmetic.
// variant: a compiled occupancy variant, 0 .. stage_variants(fp32)-1.
cudaError_t launch_stage(const StageArgs& a, int mode, bool visc, bool fp32, int variant, cudaStream_t s);
int stage_variants(bool fp32, bool hybrid);
// Raise the dynamic shared-memory limits of every stage kernel of the precision,
// once per process, outside any stream capture: returns when they are raised,
// whichever thread does it, and is tried again after a failure.
cudaError_t stage_prepare();
cudaError_t stage32_prepare();
cudaError_t raise_smem(const void* const* kernels, int n, size_t bytes);
// The FP32 kernels (stage32.cu); variant 0: registers for 2 CTAs per SM, else 3.
cudaError_t launch_stage32(const StageArgs& a, int mode, bool visc, int variant, cudaStream_t s);
cudaError_t launch_stage32_batched(const BatchStage& b, int mode, bool visc, bool hybrid, cudaStream_t s);
// Hybrid: evaluate the listed faces (the widening pass's lists; every face
// while force_weno is set) into a.wflux, where the stage kernel reads them:
// before each hybrid stage-kernel launch, on the same input.
cudaError_t launch_weno_faces(const StageArgs& a, int mode, long nfaces, const int2* list, cudaStream_t s);
// Size the evaluation kernel's grid (once, outside any stream capture).
cudaError_t weno_prepare();
// modes 1..3 only; hybrid: the StageArgs carry decision masks.
cudaError_t launch_stage_batched(const BatchStage& b, int mode, bool visc, bool fp32, bool hybrid, cudaStream_t s);
constexpr int STAGE_TI = kTileI, STAGE_TJ = kTileJ;  // columns of a CTA's tile
void stage_tiles(const Dims& d, int* ntile_i, int* ntile_j);

}  // namespace cbns
