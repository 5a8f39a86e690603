// Host-side partition of a block's (j, k) line plane into the tiles of the
// tile wavefront sweeps (sweep_tiles.cuh), and the sizes of their arrays.
#pragma once
#include <algorithm>
#include <cstddef>
#include <vector>

namespace orion {

// Lines per tile at most.  FP32 tiles of 112 run two to an SM, FP64 tiles of 96
// keep their waves in 227 KB of shared memory.  An FP64 case with few lines
// takes tiles of 64: it has SMs to spare, and a wave of two warps is shorter
// than one of three (they share the SM's load path).  Few: at most 148 x 64
// grid lines along i in all blocks, one small tile on each of a B200's SMs (97x49x33 by stages
// 5.29 ms against 5.71, Euler 111x53x47 3.97 against 4.15; 193x97x65, 12,936
// lines, 2.63 against 2.54; FP32 gained nothing).
constexpr int kTileLinesSmall = 64;
constexpr long long kTileSmallCase = 148 * kTileLinesSmall;
constexpr int tile_max_lines(size_t ssz, bool small) { return ssz == 8 ? (small ? kTileLinesSmall : 96) : 112; }
constexpr int kTileMaxEdge = 32;    // jw + kh (one halo warp)
// Components of the hyperplane form's point arrays.  The two forms' arrays
// share memory (only the form in use keeps its arrays), so a plan that needs
// no more than these costs a case no device memory.
constexpr int kPlaneComps = 72;

struct TilePlan {
  std::vector<int> jb, kb;       // tile bounds: column a holds j in [jb[a], jb[a+1])
  std::vector<long long> base;   // slot of tile (a, b)'s wave 0, line 0 at base[b * nJ + a]
  std::vector<long long> ej, ek; // first edge record shared with tile (a+1, b) / (a, b+1)
  long long slots = 0, records = 0;
  int nJ() const { return (int)jb.size() - 1; }
  int nK() const { return (int)kb.size() - 1; }
  int jw(int a) const { return jb[a + 1] - jb[a]; }
  int kh(int b) const { return kb[b + 1] - kb[b]; }
};

struct TileBytes {
  size_t own, nb, rec;  // per slot (own operands, neighbour state) and per edge record
};
inline TileBytes tile_bytes(size_t ssz) { return ssz == 8 ? TileBytes{176, 128, 64} : TileBytes{80, 48, 32}; }

// Bytes of a block's tile arrays, each 256-byte aligned.
inline size_t tile_array_bytes(long long slots, long long records, size_t ssz) {
  const TileBytes t = tile_bytes(ssz);
  auto up = [](size_t x) { return (x + 255) / 256 * 256; };
  return up(t.own * (size_t)slots) + up(t.nb * (size_t)slots) + up(t.rec * (size_t)records);
}

// Slots and edge records of the even partition into nJ x nK tiles.
inline void tile_counts(int ni, int nj, int nk, int nJ, int nK, long long& slots, long long& records) {
  // sum over the tiles of (ni + jw + kh) jw kh: every wave, and a wave of zeros
  // before the first and after the last; widths are n / p or one more
  auto squares = [](long long n, long long p) { return p * (n / p) * (n / p) + (n % p) * (2 * (n / p) + 1); };
  slots = (long long)ni * nj * nk + nk * squares(nj, nJ) + nj * squares(nk, nK);
  records = (long long)ni * nk * (nJ - 1) + (long long)ni * nj * (nK - 1);
}

// The even partition with the least work in waves: tiles x warps (a halo pair
// counted with the compute warps) x waves, weighted by the hops the wavefront
// takes through the tiles.  Partitions whose arrays outgrow the hyperplane
// form's are taken only when none fits.
inline TilePlan make_tile_plan(int ni, int nj, int nk, size_t ssz, int max_lines) {
  const size_t budget = (size_t)kPlaneComps * ssz * (size_t)ni * nj * nk;
  int bJ = nj, bK = nk;
  double best = -1.0;
  size_t least = 0;
  bool fits = false;
  int lastJ = 0;
  for (int w = kTileMaxEdge - 1; w >= 1; --w) {
    const int nJ = (nj + w - 1) / w;
    if (nJ == lastJ) continue;
    lastJ = nJ;
    const int jw = (nj + nJ - 1) / nJ;
    int lastK = 0;
    for (int h = std::min(kTileMaxEdge - jw, max_lines / jw); h >= 1; --h) {
      const int nK = (nk + h - 1) / h;
      if (nK == lastK) continue;
      lastK = nK;
      const int kh = (nk + nK - 1) / nK;
      long long slots, records;
      tile_counts(ni, nj, nk, nJ, nK, slots, records);
      const size_t bytes = tile_array_bytes(slots, records, ssz);
      const bool ok = bytes <= budget;
      const double warps = (jw * kh + 31) / 32 + 1.0;
      const double cost = (double)nJ * nK * warps * (ni + jw + kh - 2) *
                          (1.0 + 2.0 * (nJ + nK) / (double)(ni + nj + nk));
      const bool better = ok ? (!fits || cost < best) : (!fits && (best < 0.0 || bytes < least));
      if (better) {
        best = cost;
        least = bytes;
        fits = ok;
        bJ = nJ;
        bK = nK;
      }
    }
  }
  TilePlan p;
  for (int a = 0; a <= bJ; ++a) p.jb.push_back((int)((long long)a * nj / bJ));
  for (int b = 0; b <= bK; ++b) p.kb.push_back((int)((long long)b * nk / bK));
  p.base.resize((size_t)bJ * bK);
  p.ej.assign((size_t)bJ * bK, 0);
  p.ek.assign((size_t)bJ * bK, 0);
  for (int b = 0; b < bK; ++b)
    for (int a = 0; a < bJ; ++a) {
      const size_t t = (size_t)b * bJ + a;
      const long long lines = (long long)p.jw(a) * p.kh(b);
      p.base[t] = p.slots + lines;
      p.slots += (ni + p.jw(a) + p.kh(b)) * lines;
      if (a + 1 < bJ) {
        p.ej[t] = p.records;
        p.records += (long long)ni * p.kh(b);
      }
      if (b + 1 < bK) {
        p.ek[t] = p.records;
        p.records += (long long)ni * p.jw(a);
      }
    }
  return p;
}

}  // namespace orion
