// Checks the tile partition of the tile wavefront sweeps (tile_plan.hpp) for
// blocks of the given sizes, with the kernel's own address arithmetic
// (sweep_tiles.cuh): every point has one slot of its own in range; a halo
// line's point has the slot its owner gives it; both sides of an edge record
// name the same record, each record has one point; the tiles a tile waits for
// start earlier; a wave of zeros lies before and after a tile's.
// Usage: plan_check ni nj nk [ni nj nk ...]; prints "ok" or the first fault.
#include <cstdio>
#include <cstdlib>
#include <map>
#include <string>

#include "tile_plan.hpp"

using namespace orion;

static int fault(const char* what, int ni, int nj, int nk, size_t ssz) {
  std::printf("%s: %d x %d x %d, %zu-byte fields\n", what, ni, nj, nk, ssz);
  return 1;
}

static int check(int ni, int nj, int nk, size_t ssz, int max_lines) {
  const TilePlan p = make_tile_plan(ni, nj, nk, ssz, max_lines);
  const int nJ = p.nJ(), nK = p.nK();
  if (p.jb.front() != 0 || p.jb.back() != nj || p.kb.front() != 0 || p.kb.back() != nk) return fault("cover", ni, nj, nk, ssz);
  if (tile_array_bytes(p.slots, p.records, ssz) > (size_t)kPlaneComps * ssz * ni * nj * nk) return fault("memory", ni, nj, nk, ssz);
  auto col = [&](int j) { int a = 0; while (p.jb[a + 1] <= j) ++a; return a; };
  auto row = [&](int k) { int b = 0; while (p.kb[b + 1] <= k) ++b; return b; };
  auto slot = [&](int i, int j, int k) {  // tile_slot()
    const int a = col(j), b = row(k), tj = j - p.jb[a], tk = k - p.kb[b];
    return p.base[(size_t)b * nJ + a] + (long long)(i + tj + tk) * (p.jw(a) * p.kh(b)) + tk * p.jw(a) + tj;
  };
  {  // the closed form the plan was chosen by
    long long slots, records;
    tile_counts(ni, nj, nk, nJ, nK, slots, records);
    if (slots != p.slots || records != p.records) return fault("counts", ni, nj, nk, ssz);
  }
  std::vector<char> seen((size_t)p.slots, 0);
  for (int k = 0; k < nk; ++k)
    for (int j = 0; j < nj; ++j)
      for (int i = 0; i < ni; ++i) {
        const long long g = slot(i, j, k);
        if (g < 0 || g >= p.slots || seen[(size_t)g]++) return fault("slot", ni, nj, nk, ssz);
      }
  std::vector<char> rec((size_t)p.records + 1, 0);
  for (int b = 0; b < nK; ++b)
    for (int a = 0; a < nJ; ++a) {
      const int jw = p.jw(a), kh = p.kh(b), nsteps = ni + jw + kh - 2;
      const size_t t = (size_t)b * nJ + a;
      if (jw < 1 || kh < 1 || jw * kh > max_lines || jw + kh > kTileMaxEdge) return fault("tile size", ni, nj, nk, ssz);
      if (p.base[t] < jw * kh || p.base[t] + (long long)(nsteps + 1) * jw * kh > p.slots) return fault("waves", ni, nj, nk, ssz);
      for (int dir = 1; dir >= -1; dir -= 2) {
        // own lines: point and slot by step
        for (int l = 0; l < jw * kh; ++l) {
          const int tk = l / jw, tj = l - tk * jw;
          for (int s = 0; s < nsteps; ++s) {
            const int w = dir > 0 ? s : nsteps - 1 - s, i = w - tj - tk;
            if (i < 0 || i >= ni) continue;
            if (p.base[t] + (long long)w * (jw * kh) + l != slot(i, p.jb[a] + tj, p.kb[b] + tk)) return fault("own slot", ni, nj, nk, ssz);
          }
        }
        for (int side = 0; side < 2; ++side)  // halo lines below (0) and above (1)
          for (int lane = 0; lane < jw + kh; ++lane) {
            const bool isj = lane < kh;
            const int q = isj ? lane : lane - kh;
            if (isj ? (side ? a + 1 >= nJ : a == 0) : (side ? b + 1 >= nK : b == 0)) continue;
            const int tj = isj ? (side ? jw : -1) : q, tk = isj ? q : (side ? kh : -1);
            const size_t ot = isj ? (side ? t + 1 : t - 1) : (side ? t + nJ : t - nJ);
            const int ow = isj ? p.jw(side ? a + 1 : a - 1) : jw, oh = isj ? kh : p.kh(side ? b + 1 : b - 1);
            const int oj = isj ? (side ? 0 : ow - 1) : q, ok = isj ? q : (side ? 0 : oh - 1);
            const bool behind = (side == 0) == (dir > 0);
            int met = 0;
            for (int s = -1; s <= nsteps; ++s) {
              const int w = dir > 0 ? s : nsteps - 1 - s, i = w - tj - tk;
              if (i < 0 || i >= ni) continue;
              ++met;
              if (behind && (s < -1 || s > nsteps - 1)) return fault("halo step", ni, nj, nk, ssz);
              if (!behind && s < 1) return fault("ahead step", ni, nj, nk, ssz);
              const long long g = p.base[ot] + (long long)(i + oj + ok) * (ow * oh) + ok * ow + oj;
              if (g != slot(i, p.jb[a] + tj, p.kb[b] + tk)) return fault("halo slot", ni, nj, nk, ssz);
              if (behind && dir > 0) {  // consumer's record, and the producer's for the same point
                const long long r = isj ? p.ej[t - 1] + q + (long long)i * kh : p.ek[t - nJ] + q + (long long)i * jw;
                if (r < 0 || r >= p.records || rec[(size_t)r]++) return fault("edge record", ni, nj, nk, ssz);
                const long long o = isj ? p.ej[ot] + ok + (long long)i * kh : p.ek[ot] + oj + (long long)i * jw;
                if (r != o) return fault("edge sides", ni, nj, nk, ssz);
              }
            }
            if (met != ni) return fault("halo points", ni, nj, nk, ssz);
          }
        // the tiles behind start earlier in ticket order
        auto start = [&](int x, int y) { return dir > 0 ? p.jb[x] + p.kb[y] : (nj - p.jb[x + 1]) + (nk - p.kb[y + 1]); };
        const int x = a - dir, y = b - dir;
        if ((x >= 0 && x < nJ && start(x, b) >= start(a, b)) || (y >= 0 && y < nK && start(a, y) >= start(a, b)))
          return fault("order", ni, nj, nk, ssz);
      }
    }
  return 0;
}

int main(int argc, char** argv) {
  for (int x = 1; x + 2 < argc; x += 3)
    for (size_t ssz : {4, 8})
      for (bool small : {false, true})
        if (check(std::atoi(argv[x]), std::atoi(argv[x + 1]), std::atoi(argv[x + 2]), ssz, tile_max_lines(ssz, small))) return 1;
  std::printf("ok\n");
  return 0;
}
