// Tile wavefront form of the LU-SGS / symmetric Gauss-Seidel sweeps
// (StateUpdater::lusgs_sweep and gs_pr_sweep, src/solver/StateUpdater.cpp:297-445).
//
// One launch per pass.  A CTA owns a tile of jw x kh grid lines along i of one
// block, one thread per line, and walks it wave by wave: on wave
// w = i + tj + tk the thread of line (tj, tk) updates its point i (forward
// passes take the waves upwards, backward passes downwards).  A wave lies on
// one i+j+k hyperplane, so the order is the reference's lexicographic one
// exactly: a point reads its "behind" neighbours (lower i, j, k forward, upper
// backward) after they were updated in this pass and its "ahead" neighbours
// before.
//
// What bounds it.  Small cases: the length of the chain, (ni + nj + nk) waves
// per pass, so a wave has to be short: everything a wave reads is in shared
// memory before it starts, and one CTA barrier ends it (on 193x97x65 an
// instruction issues in 20-29% of the cycles, the FP64 pipe works in 23-34%;
// the first stall is that barrier).  Large cases: the waves' latency with one
// (FP64) or two CTAs an SM, and DRAM (FP32 on 385x257x129 about 4 TB/s), so each
// operand is read once per pass.  The arrays
// are laid out in the order the tile walks them (tile, wave, 16-byte piece,
// line), so a wave of a tile is one contiguous run and comes in by one bulk
// copy per array (a copy costs its issuing warp about 100 cycles whatever its
// size; one per piece made the copies the longest part of an FP32 step); the
// compute threads issue no loads from global memory.  A slot no point has (the ramps at both ends, and
// one wave beyond each) holds zeros, and so has the ring for a line outside the
// block, so the six neighbour terms are formed without a branch.
//
// Across tiles a CTA needs the fresh increments of its behind-j and behind-k
// neighbour tiles.  The producing thread stores each into an edge record as
// soon as it has it; a warp of the consuming CTA polls the record itself,
// word by word against a value no increment can have (all bits set), and puts
// the record back to empty after reading.  So a hop between tiles costs one
// L2 store and one L2 load: no fence, no progress counter, and no reset
// between passes.  The ahead neighbours' old increments are plain loads: the
// tile that owns one only overwrites it after it has received this tile's
// fresh value of the same i, which is stored after the old one was read.
//
// Tiles are claimed through a ticket counter in an order in which a tile's
// behind tiles come first, so a CTA only ever waits on CTAs that are already
// running; the launch needs no co-residency.  Every wait is bounded: after
// spin_limit polls the error word is raised, every wait of the launch gives
// up, the passes finish on whatever data is there (in bounds), and the host
// reports ORION_E_TIMEOUT and empties the edge records.
#pragma once

#include <cstddef>

#include "kernels.cuh"
#include "tile_plan.hpp"

namespace orion {

// 16-byte pieces per point of the tile layout (tl_own: met, dyn; tl_nb: nb), FP32 / FP64:
//   met  {kx ky kz |k|} per direction                     / {kx ky}{kz |k|} per direction, {1/|k| x 2}{1/|k| -}
//   dyn  {coed r0 r1 r2}{r3 r4 - -}                       / {coed r0}{r1 r2}{r3 r4}
//   nb   {u v w H}{c visc af dq4}{dq0..3}                 / {u v}{w H}{c^2 af}{c visc}{1/2c^2 1/2c}{dq0 dq1}{dq2 dq3}{dq4 -}
//
// `ring` waves of nb are kept in shared memory: at step t waves t-1 (behind) to
// t+1 (ahead) are in use and waves up to t + ring - 2 on their way; own
// operands (met, dyn) of waves t to t + ring - 2.  FP32: six waves and two CTAs
// an SM (193x97x65, 8 blocks: 1.93 ms a step, five waves 1.98; eight waves and
// one CTA an SM the same, and 4% slower on 385x257x129).
#ifndef ORION_TILE_RING_F32
#define ORION_TILE_RING_F32 6
#endif
#ifndef ORION_TILE_RING_F64
#define ORION_TILE_RING_F64 5
#endif
template <typename T> struct TileLayout;
template <> struct TileLayout<float> {
  static constexpr int met = 3, dyn = 2, nb = 3, nb_static = 2, own = met + dyn, rec = 8, minb = 2, ring = ORION_TILE_RING_F32;
  using vec = float4;
  static constexpr bool split = false;
};
// split: on the GS passes a second set of compute warps forms the terms of the
// ahead neighbours one step early (they are known before the pass), so a step's
// chain is three terms long in place of six and the FP64 pipe has twice the
// warps.
template <> struct TileLayout<double> {
  static constexpr int met = 8, dyn = 3, nb = 8, nb_static = 5, own = met + dyn, rec = 8, minb = 1, ring = ORION_TILE_RING_F64;
  using vec = double2;
  static constexpr bool split = true;
};
// Values a point's ahead terms are handed over in: the three terms one by one
// where they are subtracted after the behind ones (forward), else their sum.
constexpr int kTileAheadValues = 15;

// One tile, in ticket order of one direction.
struct SweepTile {
  int block;
  int start;             // waves its first point is behind the block's first (list order)
  int jw, kh;
  int w[2];              // widths jw of the tiles at j-1 and j+1, 0: none
  int h[2];              // heights kh of the tiles at k-1 and k+1, 0: none
  int jb, kb;            // first line
  long long base;        // slot of wave 0, line 0 in the block's tile arrays
  long long base_j[2];   // of the tiles at j-1, j+1
  long long base_k[2];
  long long edge_j[2];   // first edge record shared with the tile at j-1, j+1 (kh per i)
  long long edge_k[2];   // at k-1, k+1 (jw per i)
};

// A tile's lines in k row `k` from line j, points from i (k_tile_prep).
struct TileRow {
  int block, i, j, k;
};

// Ticket and exit counters of one launch; the last CTA to leave clears both.
struct TileCtl {
  unsigned int ticket, done;
};

// Dynamic shared memory of tiles of `lines` lines at most: the ring (per wave
// [piece][line], then [piece][32 behind and 32 ahead halo lines]), the fresh
// increments of two waves ([piece][line, halo line]), the own operands
// ([piece][line]) and the ahead terms of two waves ([value][line]).
template <typename T>
constexpr size_t tile_smem_bytes(int lines) {
  using L = TileLayout<T>;
  return (size_t)(L::ring * L::nb + 2 * ((5 * sizeof(T) + 15) / 16)) * 16 * (size_t)(lines + 64) +
         (size_t)(L::ring - 1) * L::own * 16 * (size_t)lines +
         (L::split ? (size_t)2 * kTileAheadValues * sizeof(T) * (size_t)lines : 0);
}

// ---------------------------------------------------------------------------
// edge records: five increments and the empty value (all bits set).  No
// arithmetic result has that pattern except a NaN with its sign flipped, which
// the producer stores as another NaN.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void edge_store(float* r, const float v[5]) {
  unsigned b[5];
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    b[m] = __float_as_uint(v[m]);
    if (b[m] == 0xffffffffu) b[m] = 0x7fffffffu;
  }
  asm volatile("st.relaxed.gpu.global.v4.b32 [%0], {%1,%2,%3,%4};\n" ::"l"(r), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3])
               : "memory");
  asm volatile("st.relaxed.gpu.global.b32 [%0], %1;\n" ::"l"(r + 4), "r"(b[4]) : "memory");
}
__device__ __forceinline__ void edge_store(double* r, const double v[5]) {
  unsigned long long b[5];
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    b[m] = (unsigned long long)__double_as_longlong(v[m]);
    if (b[m] == ~0ull) b[m] = 0x7fffffffffffffffull;
  }
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1,%2};\n" ::"l"(r), "l"(b[0]), "l"(b[1]) : "memory");
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1,%2};\n" ::"l"(r + 2), "l"(b[2]), "l"(b[3]) : "memory");
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;\n" ::"l"(r + 4), "l"(b[4]) : "memory");
}
__device__ __forceinline__ void edge_load(const float* r, unsigned b[5]) {
  asm volatile("ld.relaxed.gpu.global.v4.b32 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3])
               : "l"(r)
               : "memory");
  asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];\n" : "=r"(b[4]) : "l"(r + 4) : "memory");
}
__device__ __forceinline__ void edge_load(const double* r, unsigned long long b[5]) {
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0,%1}, [%2];\n" : "=l"(b[0]), "=l"(b[1]) : "l"(r) : "memory");
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0,%1}, [%2];\n" : "=l"(b[2]), "=l"(b[3]) : "l"(r + 2) : "memory");
  asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];\n" : "=l"(b[4]) : "l"(r + 4) : "memory");
}
__device__ __forceinline__ void edge_clear(float* r) {
  asm volatile("st.relaxed.gpu.global.v4.b32 [%0], {%1,%1,%1,%1};\n" ::"l"(r), "r"(0xffffffffu) : "memory");
  asm volatile("st.relaxed.gpu.global.b32 [%0], %1;\n" ::"l"(r + 4), "r"(0xffffffffu) : "memory");
}
__device__ __forceinline__ void edge_clear(double* r) {
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1,%1};\n" ::"l"(r), "l"(~0ull) : "memory");
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1,%1};\n" ::"l"(r + 2), "l"(~0ull) : "memory");
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;\n" ::"l"(r + 4), "l"(~0ull) : "memory");
}
template <typename T> struct EdgeBits;
template <> struct EdgeBits<float> { using type = unsigned; };
template <> struct EdgeBits<double> { using type = unsigned long long; };
template <typename U>
__device__ __forceinline__ bool edge_full(const U b[5]) {
  const U e = ~U(0);
  return b[0] != e && b[1] != e && b[2] != e && b[3] != e && b[4] != e;
}

// mbarrier of one ring wave: one arrival (the copying warp's, with the wave's
// byte count), completed by the bulk copies.
__device__ __forceinline__ void mbar_init(unsigned long long* m) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"((unsigned)__cvta_generic_to_shared(m)) : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned long long* m, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"((unsigned)__cvta_generic_to_shared(m)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try(unsigned m, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(m), "r"(parity)
      : "memory");
  return ok != 0;
}
// A copy of this CTA's own always arrives; the bound is there all the same.
__device__ __forceinline__ void mbar_wait(unsigned m, unsigned parity, int* err) {
  for (int it = 0; !mbar_try(m, parity); ++it)
    if (it > (1 << 24)) {
      sweep_gave_up(err);
      return;
    }
}
__device__ __forceinline__ void bulk_copy(void* smem, const void* gmem, unsigned bytes, unsigned long long* m) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                   (unsigned)__cvta_generic_to_shared(smem)),
               "l"(gmem), "r"(bytes), "r"((unsigned)__cvta_generic_to_shared(m))
               : "memory");
}

// ---------------------------------------------------------------------------
// one point's own operands and one neighbour's term, per precision; all
// operands in shared memory
// ---------------------------------------------------------------------------
template <typename T, int MODE> struct TilePoint;

// FP32 (mixed path).  With the neighbour's spectral radius taken through this
// point's metric k, the split eigenvalues of compute_flux_splitting
// (StateUpdater.cpp:217-265) give 2 l1 - l4 - l5 = 0 and l4 - l5 = 2 c |k|
// identically, so x1 = 0, x2 = |k| / 2 and every 1/|k| cancels:
//   2 fs0 = a d0 - D,  2 fsm = a dm + km dh - um D,  2 fs4 = a d4 + ct dh - H D
// with ct = k.u, D = ct d0 - k.d, dh = af d0 - (gamma-1)(u.d - d4) and
// a = ct +- (|ct| + c |k| + visc |k|^2) carrying the viscous radius too.  About
// 30 operations a neighbour and no division, against 70 with the coefficients
// formed one by one; the rounding noise of x1 is gone.
template <int MODE>
struct TilePoint<float, MODE> {
  float4 m[3];
  float4 y0;  // coed and rhs 0..2
  float2 y1;  // rhs 3, 4
  // own operands of a wave ([piece][nl]); in the backward LU-SGS pass the
  // forward increment, from the wave's ring plane, takes the RHS's place
  __device__ __forceinline__ void load(const uint4* own, int nl, int l, const uint4* plane) {
    const float4* const p = reinterpret_cast<const float4*>(own) + l;
#pragma unroll
    for (int d = 0; d < 3; ++d) m[d] = p[d * nl];
    if (MODE == SW_LUSGS_BWD) {
      const float4* const q = reinterpret_cast<const float4*>(plane) + l;
      y0 = q[2 * nl];
      y1.x = reinterpret_cast<const float*>(q + nl)[3];
      y1.y = reinterpret_cast<const float*>(p + 3 * nl)[0];
    } else {
      y0 = p[3 * nl];
      y1 = *reinterpret_cast<const float2*>(p + 4 * nl);
    }
  }
  // neighbour across direction d, lower or upper: its first ring piece (ps
  // apart), and its fresh increment, or the ring's old one
  template <bool FRESH>
  __device__ __forceinline__ void term(int d, bool upper, const uint4* first, int ps, const uint4* fresh, int sl, int slot,
                                       float g1, int, float acc[5]) const {
    const float4* p = reinterpret_cast<const float4*>(first);
    const float4 A = p[0];
    float4 B = p[ps], D;
    if (FRESH) {
      D = reinterpret_cast<const float4*>(fresh)[slot];
      B.w = reinterpret_cast<const float*>(fresh + sl)[slot];
    } else {
      D = p[2 * ps];
    }
    const float4 k = m[d];
    const float ct = k.x * A.x + k.y * A.y + k.z * A.z;
    const float rr = fabsf(ct) + B.x * k.w, vr = B.y * (k.w * k.w);
    const float a = upper ? (MODE == SW_GS ? ct - (rr + vr) : ct - rr + vr) : ct + (rr + vr);
    const float kd = k.x * D.y + k.y * D.z + k.z * D.w;
    const float DC = ct * D.x - kd;
    const float dh = B.z * D.x - g1 * (A.x * D.y + A.y * D.z + A.z * D.w - B.w);
    const float s = (MODE == SW_GS && upper) ? -1.f : 1.f;
    acc[0] += s * (a * D.x - DC);
    acc[1] += s * (a * D.y + k.x * dh - A.x * DC);
    acc[2] += s * (a * D.z + k.y * dh - A.y * DC);
    acc[3] += s * (a * D.w + k.z * dh - A.z * DC);
    acc[4] += s * (a * B.w + ct * dh - A.w * DC);
  }
  __device__ __forceinline__ void result(const float acc[5], float v[5]) const {
    if (MODE == SW_LUSGS_BWD) {
      const float h = 0.5f * y1.y;
      v[0] = y0.x - acc[0] * h;
      v[1] = y0.y - acc[1] * h;
      v[2] = y0.z - acc[2] * h;
      v[3] = y0.w - acc[3] * h;
      v[4] = y1.x - acc[4] * h;
    } else {
      v[0] = (0.5f * acc[0] - y0.y) * y0.x;
      v[1] = (0.5f * acc[1] - y0.z) * y0.x;
      v[2] = (0.5f * acc[2] - y0.w) * y0.x;
      v[3] = (0.5f * acc[3] - y1.x) * y0.x;
      v[4] = (0.5f * acc[4] - y1.y) * y0.x;
    }
  }
  static __device__ __forceinline__ void fresh_store(uint4* fresh, int sl, int slot, const float v[5]) {
    reinterpret_cast<float4*>(fresh)[slot] = make_float4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<float*>(fresh + sl)[slot] = v[4];
  }
  // p: the point's first nb piece, pieces cs bytes apart
  static __device__ __forceinline__ void store(char* p, int cs, const float v[5]) {
    *reinterpret_cast<float4*>(p + 2 * cs) = make_float4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<float*>(p + cs)[3] = v[4];
  }
};

// FP64 (plain path): the reference's operations in the reference's order; the
// two divisions of the pair's coefficients share the reciprocals prepared once
// per point.
template <int MODE>
struct TilePoint<double, MODE> {
  double k[9], gm[3], inv[3], coed, y[5];
  __device__ __forceinline__ void load(const uint4* own, int nl, int l, const uint4* plane) {
    const double2* const p = reinterpret_cast<const double2*>(own) + l;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double2 a = p[2 * d * nl], b = p[(2 * d + 1) * nl];
      k[3 * d] = a.x;
      k[3 * d + 1] = a.y;
      k[3 * d + 2] = b.x;
      gm[d] = b.y;
    }
    const double2 a = p[6 * nl];
    inv[0] = a.x;
    inv[1] = a.y;
    inv[2] = reinterpret_cast<const double*>(p + 7 * nl)[0];
    if (MODE == SW_LUSGS_BWD) {
      coed = reinterpret_cast<const double*>(p + 8 * nl)[0];
      const double2* const q = reinterpret_cast<const double2*>(plane) + l;
      const double2 e = q[5 * nl], h = q[6 * nl];
      y[0] = e.x;
      y[1] = e.y;
      y[2] = h.x;
      y[3] = h.y;
      y[4] = reinterpret_cast<const double*>(q + 7 * nl)[0];
    } else {
      const double2 e = p[8 * nl], h = p[9 * nl], w = p[10 * nl];
      coed = e.x;
      y[0] = e.y;
      y[1] = h.x;
      y[2] = h.y;
      y[3] = w.x;
      y[4] = w.y;
    }
  }
  template <bool FRESH>
  __device__ __forceinline__ void term(int d, bool upper, const uint4* first, int ps, const uint4* fresh, int sl, int slot,
                                       double g1, int nvis, double acc[5]) const {
    const double2* p = reinterpret_cast<const double2*>(first);
    const double2 uv = p[0], wh = p[ps], ca = p[2 * ps], cv = p[3 * ps], rc = p[4 * ps];
    const double2* f = FRESH ? reinterpret_cast<const double2*>(fresh) + slot : p + 5 * ps;
    const int fs = FRESH ? sl : ps;
    const double2 d01 = f[0], d23 = f[fs];
    const double dn[5] = {d01.x, d01.y, d23.x, d23.y,
                          FRESH ? reinterpret_cast<const double*>(fresh + 2 * sl)[slot]
                                : reinterpret_cast<const double*>(f + 2 * fs)[0]};
    const double nq[6] = {uv.x, uv.y, wh.x, wh.y, ca.x, ca.y};
    const double kx = k[3 * d], ky = k[3 * d + 1], kz = k[3 * d + 2];
    const double c2 = ca.x, cm = cv.x;
    // the neighbour's state as seen through this point's metric: spectral
    // radius, split eigenvalues and viscous radius (calc_spectral_radius,
    // compute_flux_splitting, calc_visc_spectral_radius,
    // StateUpdater.cpp:175-265)
    const double ct = uv.x * kx + uv.y * ky + wh.x * kz + 0.0;
    const double r = fabs(ct) + cm * gm[d];
    const double gmc = gm[d] < 1.0e-30 ? 1.0e-30 : gm[d];
    const double sr = upper ? -r : r;
    double l1 = ct, l4 = ct + cm * gmc, l5 = ct - cm * gmc;
    l1 = 0.5 * (l1 + sr);
    l4 = 0.5 * (l4 + sr);
    l5 = 0.5 * (l5 + sr);
    double pc[5], nrm[3];
    pc[0] = l1;
    pc[1] = quotient(2.0 * l1 - l4 - l5, 2.0 * c2, rc.x);
    pc[2] = quotient(l4 - l5, 2.0 * cm, rc.y);
    pc[3] = ct * inv[d];
    pc[4] = nvis == 1 ? 0.5 * (cv.y * (kx * kx + ky * ky + kz * kz)) : 0.0;
    nrm[0] = kx * inv[d];
    nrm[1] = ky * inv[d];
    nrm[2] = kz * inv[d];
    split_term<double, MODE>(upper ? 3 : 0, g1, nvis, dn, nq, pc, nrm, acc);
  }
  __device__ __forceinline__ void result(const double acc[5], double v[5]) const {
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      if (MODE == SW_LUSGS_BWD) v[m] = y[m] - acc[m] * coed;
      else if (MODE == SW_LUSGS_FWD) v[m] = (-y[m] + acc[m]) * coed;
      else v[m] = (acc[m] + -y[m]) * coed;
    }
  }
  static __device__ __forceinline__ void fresh_store(uint4* fresh, int sl, int slot, const double v[5]) {
    reinterpret_cast<double2*>(fresh)[slot] = make_double2(v[0], v[1]);
    reinterpret_cast<double2*>(fresh + sl)[slot] = make_double2(v[2], v[3]);
    reinterpret_cast<double*>(fresh + 2 * sl)[slot] = v[4];
  }
  static __device__ __forceinline__ void store(char* p, int cs, const double v[5]) {
    *reinterpret_cast<double2*>(p + 5 * cs) = make_double2(v[0], v[1]);
    *reinterpret_cast<double2*>(p + 6 * cs) = make_double2(v[2], v[3]);
    *reinterpret_cast<double*>(p + 7 * cs) = v[4];
  }
};

// MODE: SW_LUSGS_FWD (lower neighbours), SW_LUSGS_BWD (upper), SW_GS with DIR
// +1 / -1 (all six).  Warps: TT compute threads, one a line (split GS passes: TT
// more for the ahead terms), one warp for the behind halo lines, and one that
// starts the bulk copies and, on the GS passes, brings the ahead halo lines.
//
// Step t handles wave t (forward) or W-1-t.  At its start wave t + FN is sent
// for; the compute threads wait for wave t+1, update wave t from ring waves
// t-1 and t+1 and the fresh increments of t-1; the behind warp delivers its
// lines' fresh increments of wave t (read at t+1).
template <typename S, typename T, int MODE, int DIR, int TT>
__global__ void __launch_bounds__(TT * (MODE == SW_GS && TileLayout<T>::split ? 2 : 1) + 64, TileLayout<T>::minb)
    k_sweep_tiles(const BlockDev<S>* __restrict__ blocks, const SweepTile* __restrict__ tiles, int ntiles, int lines,
                  TileCtl* __restrict__ ctl, int* __restrict__ err, long long spin_limit) {
  static_assert(sizeof(S) == sizeof(T), "the tile sweeps keep operands in their storage precision");
  using L = TileLayout<T>;
  using U = typename EdgeBits<T>::type;
  constexpr int R = L::ring, NB = L::nb, FN = R - 2;
  constexpr bool SPLIT = MODE == SW_GS && L::split;
  constexpr int NC = TT / 32 * (SPLIT ? 2 : 1);    // compute warps
  constexpr int LAND = SPLIT ? FN - 3 : FN - 2;    // copies that may be on their way: waves to t + 2 (split: t + 3) are in
  static_assert(LAND >= 0, "the split passes look one wave further");
  // own pieces copied (the last of the run stay: the backward LU-SGS pass reads no RHS)
  constexpr int OWN = L::met + (MODE == SW_LUSGS_BWD ? 1 : L::dyn);
  constexpr bool LOWER = MODE != SW_LUSGS_BWD, UPPER = MODE != SW_LUSGS_FWD;
  constexpr int FP = (5 * (int)sizeof(T) + 15) / 16;  // 16-byte units of a slot's fresh increment
  extern __shared__ __align__(128) uint4 ring[];      // R planes, fresh [2][FP][sl], own [R - 1][own][lines]
  __shared__ unsigned long long s_full[R];
  __shared__ int s_slot;
  const int sl = lines + 64;
  const int plane = NB * sl, fplane = FP * sl, oplane = L::own * lines;
  uint4* const fresh = ring + R * plane;
  uint4* const own = fresh + 2 * fplane;
  T* const ahead_terms = reinterpret_cast<T*>(own + (R - 1) * oplane);  // [2][kTileAheadValues][lines]
  if (threadIdx.x == 0) {
    s_slot = (int)atomicAdd(&ctl->ticket, 1u);
#pragma unroll
    for (int r = 0; r < R; ++r) mbar_init(&s_full[r]);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  // zeros where nothing is ever copied: halo lines outside the block (the last
  // NB x 64 of a plane), and the wave before the first (ring plane R - 1, fresh
  // plane 1)
  for (int x = threadIdx.x; x < R * NB * 64; x += blockDim.x)
    ring[x / (NB * 64) * plane + NB * lines + x % (NB * 64)] = make_uint4(0, 0, 0, 0);
  for (int x = threadIdx.x; x < plane; x += blockDim.x) ring[(R - 1) * plane + x] = make_uint4(0, 0, 0, 0);
  for (int x = threadIdx.x; x < 2 * fplane; x += blockDim.x) fresh[x] = make_uint4(0, 0, 0, 0);
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");  // before the bulk copies that reuse plane R - 1
  __syncthreads();
  const SweepTile W = tiles[s_slot];
  const BlockDev<S>& B = blocks[W.block];
  const int ni = B.ni, jw = W.jw, kh = W.kh, nl = jw * kh;
  const int nsteps = ni + jw + kh - 2;
  char* const nb = B.tl_nb;
  T* const edge = reinterpret_cast<T*>(B.tl_edge);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (warp < NC) {
    // ------------------------- compute threads -------------------------
    const bool helper = SPLIT && warp >= TT / 32;
    const int l = (int)threadIdx.x - (helper ? TT : 0);
    const bool line = l < nl;
    const int tk = l / jw, tj = l - tk * jw;
    const T g1 = T(B.prm.gamma) - T(1);
    const int nvis = B.prm.nvis;
    // the j and k neighbours' lines, in the tile or among the halo lines of
    // that side: fresh slot, first ring piece in a plane, piece stride
    constexpr int HL = DIR > 0 ? 0 : 32, HU = DIR > 0 ? 32 : 0;
    struct Near {
      int slot, at, ps;
    };
    auto near = [&](bool in, int ln, int halo) {
      return in ? Near{ln, ln, nl} : Near{lines + halo, NB * lines + halo, 64};
    };
    const Near jl = near(tj > 0, l - 1, HL + tk), jh = near(tj < jw - 1, l + 1, HU + tk);
    const Near kl = near(tk > 0, l - jw, HL + kh + tj), kh_ = near(tk < kh - 1, l + jw, HU + kh + tj);
    int i = line ? (DIR > 0 ? 0 : nsteps - 1) - tj - tk : -(1 << 24);  // this thread's point at step t
    char* p = nb + ((W.base + (long long)(DIR > 0 ? 0 : nsteps - 1) * nl) * NB + l) * 16;
    const int ps = DIR * nl * NB * 16;
    T* out_j = nullptr;  // the records of the downstream tiles this line feeds, at point i
    T* out_k = nullptr;
    if (line) {
      constexpr int o = DIR > 0 ? 1 : 0;
      if (tj == (DIR > 0 ? jw - 1 : 0) && W.w[o] > 0) out_j = edge + (W.edge_j[o] + tk) * L::rec;
      if (tk == (DIR > 0 ? kh - 1 : 0) && W.h[o] > 0) out_k = edge + (W.edge_k[o] + tj) * L::rec;
    }
    const unsigned full0 = (unsigned)__cvta_generic_to_shared(s_full);
    const uint4 *pb = ring + (R - 1) * plane, *po = ring, *pa = ring + plane;  // waves t-1, t, t+1
    const uint4* pown = own;
    int ra = 1;           // ring index of wave t+1
    unsigned parity = 0;  // of its barrier
    auto next = [&]() {   // on to the next step
      i += DIR;
      pb = po;
      po = pa;
      pa += plane;
      if (++ra == R) {
        ra = 0;
        pa = ring;
        parity ^= 1;
      }
      pown = pown + oplane == own + (R - 1) * oplane ? own : pown + oplane;
    };
    mbar_wait(full0, 0, err);
    __syncthreads();
    if constexpr (SPLIT) {
      if (helper) {
        // step s: the terms of wave s's ahead neighbours (wave s + 1), read by
        // the other warps at step s, formed while they are at step s - 1
        for (int s = 0; s < nsteps; ++s) {
          mbar_wait(full0 + 8 * ra, parity, err);
          if ((unsigned)i < (unsigned)ni) {
            TilePoint<T, MODE> cur;
            cur.load(pown, nl, l, po);
            T* const out = ahead_terms + (s & 1) * kTileAheadValues * lines + l;
            T a[3][5] = {};
            constexpr bool U = DIR > 0;  // the ahead neighbours are the upper ones
            // upper terms are subtracted one by one after the lower ones: each is
            // handed over as 0 - term; lower ones are summed first
            T(&a1)[5] = a[U ? 1 : 0];
            T(&a2)[5] = a[U ? 2 : 0];
            const Near &nj = U ? jh : jl, &nk = U ? kh_ : kl;
            cur.template term<false>(0, U, pa + l, nl, fresh, sl, l, g1, nvis, a[0]);
            cur.template term<false>(1, U, pa + nj.at, nj.ps, fresh, sl, nj.slot, g1, nvis, a1);
            cur.template term<false>(2, U, pa + nk.at, nk.ps, fresh, sl, nk.slot, g1, nvis, a2);
#pragma unroll
            for (int m = 0; m < (U ? 15 : 5); ++m) out[m * lines] = a[m / 5][m % 5];
          }
          next();
          __syncthreads();
        }
      }
    }
    if (!helper) {
      if (SPLIT) __syncthreads();  // wave 0's ahead terms
      for (int t = 0; t < nsteps; ++t) {
        mbar_wait(full0 + 8 * ra, parity, err);
        if ((unsigned)i < (unsigned)ni) {
          const uint4* const fr = fresh + ((t + 1) & 1) * fplane;  // wave t-1's
          TilePoint<T, MODE> cur;
          cur.load(pown, nl, l, po);
          T acc[5] = {T(0), T(0), T(0), T(0), T(0)}, v[5];
          const T* const given = ahead_terms + (t & 1) * kTileAheadValues * lines + l;
          // lower neighbours first (i, j, k), then upper (i, j, k): the reference's order
          if (LOWER) {
            constexpr bool F = DIR > 0;
            if constexpr (SPLIT && !F) {
#pragma unroll
              for (int m = 0; m < 5; ++m) acc[m] = given[m * lines];
            } else {
              const uint4* const q = F ? pb : pa;
              cur.template term<F>(0, false, q + l, nl, fr, sl, l, g1, nvis, acc);
              cur.template term<F>(1, false, q + jl.at, jl.ps, fr, sl, jl.slot, g1, nvis, acc);
              cur.template term<F>(2, false, q + kl.at, kl.ps, fr, sl, kl.slot, g1, nvis, acc);
            }
          }
          if (UPPER) {
            constexpr bool F = DIR < 0;
            if constexpr (SPLIT && !F) {
#pragma unroll
              for (int m = 0; m < 15; ++m) acc[m % 5] += given[m * lines];
            } else {
              const uint4* const q = F ? pb : pa;
              cur.template term<F>(0, true, q + l, nl, fr, sl, l, g1, nvis, acc);
              cur.template term<F>(1, true, q + jh.at, jh.ps, fr, sl, jh.slot, g1, nvis, acc);
              cur.template term<F>(2, true, q + kh_.at, kh_.ps, fr, sl, kh_.slot, g1, nvis, acc);
            }
          }
          cur.result(acc, v);
          TilePoint<T, MODE>::fresh_store(fresh + (t & 1) * fplane, sl, l, v);
          if (out_j) edge_store(out_j + (long long)i * (kh * L::rec), v);
          if (out_k) edge_store(out_k + (long long)i * (jw * L::rec), v);
          TilePoint<T, MODE>::store(p, nl * 16, v);
        }
        p += ps;
        next();
        __syncthreads();
      }
    } else {
      __syncthreads();  // the last step
    }
  } else {
    // ------------------- behind / ahead halo lines ----------------------
    const bool behind = warp == NC;
    const int side = (behind == (DIR > 0)) ? 0 : 1;  // lower or upper neighbours
    const bool isj = lane < kh;
    const int q = isj ? lane : lane - kh;
    const bool on = (behind || MODE == SW_GS) && (isj ? W.w[side] > 0 : (q < jw && W.h[side] > 0));
    const int tj = isj ? (side ? jw : -1) : q, tk = isj ? q : (side ? kh : -1);
    const int halo = (behind ? 0 : 32) + lane;
    // the neighbour tile's own coordinates of this line
    const int ow = isj ? W.w[side] : jw, oh = isj ? kh : W.h[side];
    const int oj = isj ? (side ? 0 : ow - 1) : q, ok = isj ? q : (side ? 0 : oh - 1);
    const int onl = ow * oh;
    int i = on ? (DIR > 0 ? 0 : nsteps - 1) - tj - tk : -(1 << 24);  // its point on step 0
    const char* src =
        nb + (((isj ? W.base_j[side] : W.base_k[side]) + (long long)(i + oj + ok) * onl) * NB + ok * ow + oj) * 16;
    const int ss = DIR * onl * NB * 16;
    auto valid = [&](int x) { return (unsigned)x < (unsigned)ni; };
    auto fetch = [&](int r, int s) {  // the line's point s steps from now into ring index r
      if (valid(i + s * DIR)) {
        const char* g = src + s * ss;
        uint4* dst = ring + r * plane + NB * lines + halo;
#pragma unroll
        for (int c = 0; c < NB; ++c) cp_async16(dst + c * 64, g + c * onl * 16);
      }
    };
    if (!behind) {
      // a wave's bulk copies: lane 0 the neighbour state, lane 1 the own operands
      const bool own_run = lane == 1;
      const int per = own_run ? L::own : NB;
      const char* const run = (own_run ? B.tl_own : nb) + (W.base + (long long)(DIR > 0 ? 0 : nsteps - 1) * nl) * per * 16;
      uint4* const into = own_run ? own : ring;
      const int into_plane = own_run ? oplane : plane, into_ring = own_run ? R - 1 : R;
      const long long ws = (long long)DIR * nl * per * 16;
      const unsigned bytes = (unsigned)nl * 16;
      auto send = [&](int w) {  // wave w of the sweep, 0 .. nsteps (the zeros past the last)
        unsigned long long* const m = &s_full[w % R];
        if (lane == 0) mbar_expect(m, bytes * (NB + OWN));
        __syncwarp();
        if (lane < 2) bulk_copy(into + w % into_ring * into_plane, run + w * ws, bytes * (own_run ? OWN : NB), m);
      };
#pragma unroll
      for (int s = 0; s < FN; ++s) {
        send(s);
        fetch(s, s);
        cp_async_commit();
      }
      cp_async_wait<LAND>();
      __syncthreads();
      if (SPLIT) __syncthreads();  // wave 0's ahead terms
      int r = FN;  // ring index of wave t + FN
      for (int t = 0; t < nsteps; ++t) {
        if (t + FN <= nsteps) send(t + FN);
        fetch(r, FN);
        cp_async_commit();
        i += DIR;
        src += ss;
        if (++r == R) r = 0;
        cp_async_wait<LAND>();
        __syncthreads();
      }
    } else {
      // Records are asked for in pairs, two and three steps before they are due,
      // so that no step waits for an L2 load.  (In pairs: a warp's wait for a
      // load is a wait for every later load too, so asking at every step makes
      // every step as long as a load.)
      const int per = (isj ? kh : jw) * L::rec;
      const int slot = lines + halo;
      T* const rec = edge + ((isj ? W.edge_j[side] : W.edge_k[side]) + q) * L::rec;
      bool dead = false;
      U b[2][2][5];
      auto ask = [&](int x, U(&r)[2][5]) {  // reads the records of points x and x + DIR without waiting for them to fill
        if (valid(x)) edge_load(rec + (long long)x * per, r[0]);
        if (valid(x + DIR)) edge_load(rec + (long long)(x + DIR) * per, r[1]);
      };
      // fresh increments of step s's wave (the lane's point x) into fresh plane s & 1
      auto deliver = [&](int s, int x, U(&r)[5]) {
        bool full = !valid(x) || edge_full(r);
        long long it = 0;
        while (!dead && __any_sync(0xffffffffu, !full)) {
          bool stop = ++it > spin_limit;
          if ((it & 31) == 0 && *(volatile int*)err) stop = true;
          if (__any_sync(0xffffffffu, stop)) {
            if (lane == 0) sweep_gave_up(err);
            dead = true;
            break;
          }
          if (it > 8) __nanosleep(32);
          if (!full) {
            edge_load(rec + (long long)x * per, r);
            full = edge_full(r);
          }
        }
        if (valid(x)) {
          T v[5];
#pragma unroll
          for (int m = 0; m < 5; ++m) memcpy(&v[m], &r[m], sizeof(T));
          TilePoint<T, MODE>::fresh_store(fresh + (s & 1) * fplane, sl, slot, v);
          edge_clear(rec + (long long)x * per);
        }
      };
      fetch(R - 1, -1);
#pragma unroll
      for (int s = 0; s < FN; ++s) {
        fetch(s, s);
        cp_async_commit();
      }
      ask(i - DIR, b[0]);  // steps -1 and 0
      ask(i + DIR, b[1]);  // steps 1 and 2
      cp_async_wait<LAND>();
      deliver(-1, i - DIR, b[0][0]);
      __syncthreads();
      if (SPLIT) __syncthreads();
      int r = FN;
      for (int t0 = 0; t0 < nsteps; t0 += 4) {
#pragma unroll
        for (int d = 0; d < 4; ++d) {
          const int t = t0 + d;
          if (t < nsteps) {
            fetch(r, FN);
            cp_async_commit();
            deliver(t, i, b[((d + 1) / 2) & 1][(d + 1) & 1]);
            if (d & 1) ask(i + 2 * DIR, b[(d / 2) & 1]);  // steps t + 2 and t + 3
            i += DIR;
            src += ss;
            if (++r == R) r = 0;
            cp_async_wait<LAND>();
            __syncthreads();
          }
        }
      }
    }
  }
  if (threadIdx.x == 0) {
    const unsigned int n = atomicAdd(&ctl->done, 1u);
    if (n + 1 == (unsigned)ntiles) {  // every CTA has its ticket: ready for the next launch
      ctl->ticket = 0;
      ctl->done = 0;
    }
  }
}

// ---------------------------------------------------------------------------
// natural order -> tile layout
// ---------------------------------------------------------------------------
// Static operands (metrics, magnitudes), refreshed whenever the metrics are set.
template <typename S>
__global__ void k_tile_static(const BlockDev<S>* __restrict__ blocks, int b) {
  const BlockDev<S>& B = blocks[b];
  const long long np = B.npad;
  for (long long n = blockIdx.x * (long long)blockDim.x + threadIdx.x; n < B.ncomp; n += (long long)gridDim.x * blockDim.x) {
    const int n32 = (int)n, r32 = n32 / B.ni;
    const int ii = n32 - r32 * B.ni, jj = r32 % B.nj, kk = r32 / B.nj;
    const long long idx = lin(B, NG + ii, NG + jj, NG + kk);
    const TileSlot at = tile_slot(B, ii, jj, kk);
    S k[9], gm[3], inv[3];
    for (int m = 0; m < 9; ++m) k[m] = (S)B.metrics[m * np + idx];
    for (int d = 0; d < 3; ++d) {  // unit normals of compute_flux_splitting (StateUpdater.cpp:231-249)
      gm[d] = sqrt_s(k[3 * d] * k[3 * d] + k[3 * d + 1] * k[3 * d + 1] + k[3 * d + 2] * k[3 * d + 2]);
      inv[d] = S(1) / (gm[d] < S(1.0e-30) ? S(1.0e-30) : gm[d]);
    }
    using L = TileLayout<S>;
    if constexpr (sizeof(S) == 4) {
      float4* const p = at.run<float4>(B.tl_own, L::own);
      for (int d = 0; d < 3; ++d) p[d * at.nl] = make_float4(k[3 * d], k[3 * d + 1], k[3 * d + 2], gm[d]);
    } else {
      double2* const p = at.run<double2>(B.tl_own, L::own);
      for (int d = 0; d < 3; ++d) {
        p[2 * d * at.nl] = make_double2(k[3 * d], k[3 * d + 1]);
        p[(2 * d + 1) * at.nl] = make_double2(k[3 * d + 2], gm[d]);
      }
      p[6 * at.nl] = make_double2(inv[0], inv[1]);
      p[7 * at.nl] = make_double2(inv[2], 0.0);
    }
  }
}

// Per step: masked RHS, diagonal coefficient and the state a neighbour's term
// needs (k_lusgs_prep's values).  A CTA takes kPrepI points along i of a tile's
// lines in one k row: read along i, written along the lines of each wave, the
// turn made in shared memory.  What bounds it: the latency of its loads, and
// before the turn the 16-byte writes, each to a sector of its own, half full
// (385x257x129 plain 1.81 -> 1.11 ms, mixed 0.60 -> 0.57).
constexpr int kPrepI = 16;

template <typename S, typename T>
__global__ void __launch_bounds__(256, PointwiseMinBlocks<T>::n) k_tile_prep(const BlockDev<S>* __restrict__ blocks,
                                                                             const TileRow* __restrict__ rows) {
  using L = TileLayout<T>;
  using V = typename L::vec;
  constexpr int NBP = L::nb_static, PIECES = L::dyn + NBP;
  __shared__ V s_out[PIECES][256];
  const TileRow row = rows[blockIdx.x];
  const BlockDev<S>& B = blocks[row.block];
  const ParamsDev& P = B.prm;
  const long long np = B.npad;
  const int4 tj4 = __ldg(B.t_j + row.j), tk4 = __ldg(B.t_k + row.k);
  const int jw = tj4.z, nl = jw * tk4.z, ni = min(kPrepI, B.ni - row.i);
  // jw lines of kPrepI points are at most 256 x 2: tiles are at most 31 lines wide
  for (int t0 = 0; t0 < jw * kPrepI; t0 += 256) {
    const int t = t0 + threadIdx.x, i = t % kPrepI, tj = t / kPrepI;
    __syncthreads();
    if (tj < jw && i < ni) {
      const long long idx = lin(B, NG + row.i + i, NG + row.j + tj, NG + row.k);
      const bool masked = B.bcmask[idx] != 0;
      T rhs[5];
#pragma unroll
      for (int m = 0; m < 5; ++m) rhs[m] = masked ? T(0) : (T)B.dq[m * np + idx];
      const S* pr = FluxSrc<S>::prim(B);
      const T rho = (T)pr[idx], u = (T)pr[np + idx], v = (T)pr[2 * np + idx], w = (T)pr[3 * np + idx],
              p = (T)pr[4 * np + idx];
      PrepPoint<T> q;
      const S* met = FluxSrc<S>::metrics(B);
      T km[9];
#pragma unroll
      for (int m = 0; m < 9; ++m) km[m] = (T)met[m * np + idx];
      q.form(P, rho, u, v, w, p, km, (T)B.mu[idx], (T)FluxSrc<S>::vol(B)[idx], (T)B.dt[idx]);
      if constexpr (sizeof(T) == 4) {
        s_out[0][threadIdx.x] = make_float4(q.coed, rhs[0], rhs[1], rhs[2]);
        s_out[1][threadIdx.x] = make_float4(rhs[3], rhs[4], 0.f, 0.f);
        s_out[2][threadIdx.x] = make_float4(u, v, w, q.H);
        s_out[3][threadIdx.x] = make_float4(q.c, q.vcoef, q.af, 0.f);
      } else {
        s_out[0][threadIdx.x] = make_double2(q.coed, rhs[0]);
        s_out[1][threadIdx.x] = make_double2(rhs[1], rhs[2]);
        s_out[2][threadIdx.x] = make_double2(rhs[3], rhs[4]);
        s_out[3][threadIdx.x] = make_double2(u, v);
        s_out[4][threadIdx.x] = make_double2(w, q.H);
        s_out[5][threadIdx.x] = make_double2(q.c2, q.af);
        s_out[6][threadIdx.x] = make_double2(q.c, q.vcoef);
        s_out[7][threadIdx.x] = make_double2(quotient_rcp(2.0 * q.c2), quotient_rcp(2.0 * q.c));
      }
    }
    __syncthreads();
    // the lines of this pass, wave by wave: slot (i + tj) of the row's waves, consecutive lines
    const int j0 = t0 / kPrepI, jn = min(jw - j0, 256 / kPrepI);
    const long long wave = __ldg(B.t_base + tk4.x * B.tJ + tj4.x) + (long long)(row.i + tk4.y) * nl;
    for (int e = threadIdx.x; e < jn * (kPrepI + jn - 1); e += 256) {
      const int d = e / jn, x = e - d * jn, i2 = d - x;
      if (i2 < 0 || i2 >= ni) continue;
      const TileSlot at{wave + (long long)(d + j0) * nl, tk4.y * jw + j0 + x, nl};
      const int src = x * kPrepI + i2;
      V* const y = at.run<V>(B.tl_own, L::own) + L::met * nl;
      V* const z = at.run<V>(B.tl_nb, L::nb);
#pragma unroll
      for (int c = 0; c < L::dyn; ++c) y[c * nl] = s_out[c][src];
#pragma unroll
      for (int c = 0; c < NBP; ++c) z[c * nl] = s_out[L::dyn + c][src];
    }
  }
}

}  // namespace orion
