// kchunk.h - k planes per CTA of the stage kernels (host code only): the rules a
// context starts on and the candidates of cbns_autotune.
#pragma once

#include <algorithm>
#include <cmath>

namespace cbns {

constexpr int kTileI = 16, kTileJ = 15;  // columns of a CTA's tile
constexpr int kMaxChunks = 65535;        // the chunks are a launch's grid.y

// k planes per CTA of the stage kernel.  The CTAs (tiles x k chunks) run in
// waves of `slots` (SMs x CTAs per SM); a chunk costs its planes plus some
// warm-up (the ring's first planes and the first k-face), `warm` planes'
// worth.  The chunk count whose waves x (planes + warm) is least, keeping
// chunks of at least 8 planes.
inline int kchunk_by_waves(int ntiles, int nint, int slots, double warm) {
  const int maxchunk = std::max(1, nint / 8);
  double best = 1e300;
  int best_k = nint;
  for (int nchunk = 1; nchunk <= maxchunk; ++nchunk) {
    const int kc = (nint + nchunk - 1) / nchunk;
    const long items = (long)ntiles * ((nint + kc - 1) / kc);
    const long waves = (items + slots - 1) / slots;
    const double cost = (double)waves * (kc + warm);
    if (cost < best - 1e-9) {
      best = cost;
      best_k = kc;
    }
  }
  return best_k;
}

// The chunk for about `waves` waves of `slots` CTAs, chunks of at least 8 planes.
// Many short waves balance CTAs of unequal cost (tiles cut by the grid's edge,
// WENO5 faces gathered unevenly): on a 256 x 256 x 128 grid the FP64 kernel
// runs fastest at about 9 waves (13-plane chunks), 3.5% faster than at 4.6
// waves (26-plane chunks) and 10% faster than in one wave.
inline int kchunk_for_waves(int ntiles, int nint, int slots, double waves) {
  const int want = (int)std::ceil(waves * slots / ntiles);
  const int nchunk = std::max(1, std::min(want, nint / 8));
  return (nint + nchunk - 1) / nchunk;
}

// The default: about four CTAs per slot of 2 CTAs per SM, chunks of at least 8 planes.
inline int kchunk_default(int ntiles, int nint, int nsm) {
  const int nchunk = std::max(1, std::min((4 * 2 * nsm + ntiles - 1) / ntiles, nint / 8));
  return (nint + nchunk - 1) / nchunk;
}

// The chunk for a grid whose tiles at 8 planes a chunk or more make few waves of
// CTAs: the least estimate of a launch's time in planes.  A chunk takes its
// planes plus 0.7 for its start (the ring's first planes and the k-face below
// it); while the CTAs fit the slots the launch is one chunk, beyond that the
// work over the slots plus half a chunk of tail; CTAs alone on an SM run about
// 1.5 times as fast as two.  Tiles cut by the grid's edge count by their
// columns, but by half at least (a tile of few columns is not faster than that:
// with 4 columns of 240 counted as such, 4x4x5000 ran 1-plane chunks, FP64 615
// us per step, 505 with the 3 planes now chosen; split 4x4x100000 2 planes, 7754
// against 6900).  Measured us per step with this chunk against one of at least 8
// planes: FP64 64x32x16 78 against 381 (8 CTAs marched the whole block while
// 140 SMs idled), 97x61x45 245 against 272, 128x64x64 468 against 522; split
// 64x32x16 69 against 258, 97x61x45 153 against 188; hybrid (3 per SM)
// 64x32x16 146 against 277, 129x113x97 675 against 709.  Above about four
// waves the chunks stay longer: at 193x161x129 4-plane chunks take 2770 us in
// FP64 and 1618 split against 2682 and 1540 at 9.
inline int kchunk_small(int IM, int JM, int KM, int ntiles, int nsm, int per_sm) {
  const int nint = KM - 2;
  const double tiles = std::max(0.5 * ntiles, (double)(IM - 2) * (JM - 2) / (kTileI * kTileJ));
  const double slots = (double)nsm * per_sm;
  double best = 1e300;
  int best_k = nint;
  for (int kc = 1; kc <= nint; ++kc) {
    const int nchunk = (nint + kc - 1) / kc;
    if (nchunk > kMaxChunks) continue;
    const double items = (double)ntiles * nchunk, chunk = kc + 0.7;
    const double cost = items <= nsm     ? chunk / 1.5
                        : items <= slots ? chunk
                                         : (std::max(1.0, tiles * nchunk / slots) + 0.5) * chunk;
    if (cost < best - 1e-9) {
      best = cost;
      best_k = kc;
    }
  }
  return best_k;
}

// The chunk a new context starts on: about 9 waves of CTAs in FP64, with the FP32
// flux by the wave count and warm-up; where that makes fewer than four waves, the
// chunk of kchunk_small.
inline int kchunk_start(int IM, int JM, int KM, int ntiles, int nsm, bool fp32) {
  const int nint = KM - 2, per_sm = fp32 ? 3 : 2, slots = nsm * per_sm;
  int kc = fp32 ? kchunk_by_waves(ntiles, nint, slots, 0.5) : kchunk_for_waves(ntiles, nint, slots, 9.0);
  if ((long)ntiles * ((nint + kc - 1) / kc) < 4L * slots) kc = kchunk_small(IM, JM, KM, ntiles, nsm, per_sm);
  return std::max(kc, (nint + kMaxChunks - 1) / kMaxChunks);
}

}  // namespace cbns
