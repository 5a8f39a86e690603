// Kernels of the per-step path.  Each kernel cites the reference routine whose
// arithmetic it reproduces.  Templates: S = storage type of the lowered fields
// (double for the plain form, float for the mixed form), T = compute type of
// the flux / viscous / sweep arithmetic.
#pragma once
#include <cstddef>
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "device_types.cuh"
#include "numerics.cuh"

namespace orion {

// Arrays the flux kernels read: FP32 shadows on the mixed path (exactly the
// values its FP32 arithmetic converts the FP64 arrays to), the FP64 arrays on
// the plain path.
template <typename S> struct FluxSrc;
template <> struct FluxSrc<double> {
  static __device__ __forceinline__ const double* prim(const BlockDev<double>& B) { return B.prim; }
  static __device__ __forceinline__ const double* metrics(const BlockDev<double>& B) { return B.metrics; }
  static __device__ __forceinline__ const double* vol(const BlockDev<double>& B) { return B.vol; }
};
template <> struct FluxSrc<float> {
  static __device__ __forceinline__ const float* prim(const BlockDev<float>& B) { return B.prim_f; }
  static __device__ __forceinline__ const float* metrics(const BlockDev<float>& B) { return B.met_f; }
  static __device__ __forceinline__ const float* vol(const BlockDev<float>& B) { return B.vol_f; }
};


// Asynchronous copies of 16 bytes or of one value into shared memory.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned int s = (unsigned int)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }
__device__ __forceinline__ void cp_async_value(double* smem, const double* gmem) {
  const unsigned int s = (unsigned int)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_value(float* smem, const float* gmem) {
  const unsigned int s = (unsigned int)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem) : "memory");
}

template <typename S>
__device__ __forceinline__ long long lin(const BlockDev<S>& B, int i, int j, int k) {
  return (long long)i + (long long)B.nx * ((long long)j + (long long)B.ny * (long long)k);
}

template <typename S>
__device__ __forceinline__ int dim_along(const BlockDev<S>& B, int d) {
  return d == 0 ? B.ni : (d == 1 ? B.nj : B.nk);
}

template <typename S>
__device__ __forceinline__ long long stride_along(const BlockDev<S>& B, int d) {
  return d == 0 ? 1LL : (d == 1 ? (long long)B.nx : (long long)B.nx * B.ny);
}

// Memory index of along-line coordinate 0 of line `l` in direction d.  Lines
// enumerate the transverse interior coordinates, the lower one fastest.
template <typename S>
__device__ __forceinline__ long long line_origin(const BlockDev<S>& B, int d, int l) {
  if (d == 0) {
    const int jj = l % B.nj, kk = l / B.nj;
    return lin(B, 0, NG + jj, NG + kk);
  } else if (d == 1) {
    const int ii = l % B.ni, kk = l / B.ni;
    return lin(B, NG + ii, 0, NG + kk);
  }
  const int ii = l % B.ni, jj = l / B.ni;
  return lin(B, NG + ii, NG + jj, 0);
}

// ===========================================================================
// Halo copy of prim[0..4] into interface ghosts (HaloExchanger::exchange_bc,
// src/solver/HaloExchanger.cpp:70-179).  The host flattened the pack/unpack
// order into (src, dst) element offsets, last writer kept.
// ===========================================================================
static __global__ void k_halo_copy(double* __restrict__ arena, const long long* __restrict__ src,
                            const long long* __restrict__ dst, int n) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) arena[dst[t]] = arena[src[t]];
}

// The same copy for a group of cases: blockIdx.y is the member, which copies
// through its own list into its own arena (nothing is concatenated).
static __global__ void k_halo_copy_group(const GroupMember* __restrict__ members) {
  const GroupMember& M = members[blockIdx.y];
  double* const arena = M.arena;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < M.n_halo; t += gridDim.x * blockDim.x)
    arena[M.halo_dst[t]] = arena[M.halo_src[t]];
}

// ===========================================================================
// Physical BCs (src/bc/PhysicalBC.cpp:12-613).  One launch per phase; phase p
// holds the p-th physical region of every block (regions of one block are
// sequential in file order; columns of one region are independent).
// ===========================================================================
template <typename S>
__device__ __forceinline__ void bc_normal(const BlockDev<S>& B, long long idx, int s_nd, double& nx, double& ny,
                                          double& nz) {
  // get_normal (PhysicalBC.cpp:12-44)
  const int off = (s_nd - 1) * 3;
  const double mx = B.metrics[(off + 0) * B.npad + idx];
  const double my = B.metrics[(off + 1) * B.npad + idx];
  const double mz = B.metrics[(off + 2) * B.npad + idx];
  double len = sqrt(mx * mx + my * my + mz * mz);
  if (len < 1.0e-30) len = 1.0e-30;
  nx = mx / len;
  ny = my / len;
  nz = mz / len;
}

template <typename S>
__device__ __forceinline__ void dif_average(const BlockDev<S>& B, long long idx0, long long step_out) {
  // apply_dif_average (PhysicalBC.cpp:71-92): face point = mean of ghost 1 and inner 1.
  const long long ig = idx0 + step_out, ii = idx0 - step_out;
  for (int m = 0; m < 6; ++m) {
    const double vg = B.prim[m * B.npad + ig];
    const double vi = B.prim[m * B.npad + ii];
    B.prim[m * B.npad + idx0] = 0.5 * (vg + vi);
  }
}

template <typename S>
__global__ void k_bc_phase(const BlockDev<S>* __restrict__ blocks, const RegionDev* __restrict__ regions,
                           const int* __restrict__ phase_regions) {
  const RegionDev R = regions[phase_regions[blockIdx.y]];
  const int pt = blockIdx.x * blockDim.x + threadIdx.x;
  if (pt >= R.npts) return;
  const BlockDev<S> B = blocks[R.block];
  const ParamsDev& P = B.prm;
  const int wi = R.hi[0] - R.lo[0] + 1, wj = R.hi[1] - R.lo[1] + 1;
  const int i = R.lo[0] + pt % wi;
  const int j = R.lo[1] + (pt / wi) % wj;
  const int k = R.lo[2] + pt / (wi * wj);
  const long long idx0 = lin(B, i, j, k);
  const long long sd = (R.dir == 0) ? 1LL : (R.dir == 1 ? (long long)B.nx : (long long)B.nx * B.ny);
  const long long out = (R.lr == 1) ? sd : -sd;  // step from the face towards the ghosts
  const long long np = B.npad;
  double* prim = B.prim;
  auto PR = [&](int m, long long id) -> double& { return prim[m * np + id]; };

  switch (R.type) {
    case 2: {
      if (P.nvis == 1) {
        // apply_viscid_wall (PhysicalBC.cpp:254-363)
        const double gama = P.gamma, mach = P.moo;
        const double moocp = mach * mach * gama;
        const bool isothermal = (P.twall > 1.0e-6);
        const double twall_dim = (isothermal && fabs(P.tref) > 1e-16) ? P.twall / P.tref : P.twall;
        const long long i1 = idx0 - out, i2 = idx0 - 2 * out;
        const double p1 = PR(4, i1), p2 = PR(4, i2);
        double p_wall = (4.0 * p1 - p2) / 3.0;
        if (p_wall < 1.0e-6) p_wall = p1;
        double t_wall;
        if (isothermal) {
          t_wall = twall_dim;
        } else {
          const double t1 = PR(5, i1), t2 = PR(5, i2);
          t_wall = (4.0 * t1 - t2) / 3.0;
          if (t_wall < 1e-6) t_wall = t1;
        }
        const double rho_wall = moocp * p_wall / t_wall;
        for (int l = 0; l < NG; ++l) {
          const int dist = l + 1;
          const long long ig = idx0 + dist * out, ii = idx0 - dist * out;
          const double u_i = PR(1, ii), v_i = PR(2, ii), w_i = PR(3, ii);
          PR(1, ig) = -u_i;
          PR(2, ig) = -v_i;
          PR(3, ig) = -w_i;
          PR(4, ig) = PR(4, ii);
          if (isothermal) {
            const double t_inner = PR(5, ii);
            PR(5, ig) = 2.0 * t_wall - t_inner;
          } else {
            PR(5, ig) = PR(5, ii);
          }
          const double pg = PR(4, ig);
          double tg = PR(5, ig);
          if (tg < 1e-6) tg = 1.0;
          const double rho_calc = moocp * pg / tg;
          PR(0, ig) = (dist == 3) ? -rho_calc : rho_calc;
        }
        PR(0, idx0) = rho_wall;
        PR(1, idx0) = 0.0;
        PR(2, idx0) = 0.0;
        PR(3, idx0) = 0.0;
        PR(4, idx0) = p_wall;
        PR(5, idx0) = t_wall;
      } else {
        // apply_inviscid_wall (PhysicalBC.cpp:191-248)
        double nx, ny, nz;
        bc_normal(B, idx0, R.s_nd, nx, ny, nz);
        for (int l = 0; l < NG; ++l) {
          const int dist = l + 1;
          const long long ig = idx0 + dist * out, ii = idx0 - dist * out;
          const double rho_i = PR(0, ii), u_i = PR(1, ii), v_i = PR(2, ii), w_i = PR(3, ii), p_i = PR(4, ii);
          const double t_i = PR(5, ii);
          const double v_dot_n = u_i * nx + v_i * ny + w_i * nz;
          PR(0, ig) = (dist == 3) ? -rho_i : rho_i;
          PR(1, ig) = u_i - 2.0 * v_dot_n * nx;
          PR(2, ig) = v_i - 2.0 * v_dot_n * ny;
          PR(3, ig) = w_i - 2.0 * v_dot_n * nz;
          PR(4, ig) = p_i;
          PR(5, ig) = t_i;
        }
        if (P.method == 1) dif_average(B, idx0, out);
      }
      break;
    }
    case 3: {
      // apply_symmetry_bc (PhysicalBC.cpp:97-183)
      if (R.is2d) {
        for (int l = 0; l < NG; ++l) {
          const int dist = l + 1;
          const long long ig = idx0 + dist * out, ii = idx0 - dist * out;
          PR(0, ig) = PR(0, ii);
          PR(1, ig) = PR(1, ii);
          PR(2, ig) = PR(2, ii);
          PR(4, ig) = PR(4, ii);
          PR(5, ig) = PR(5, ii);
          PR(3, ig) = -PR(3, ii);
        }
      } else {
        const int im = (R.lo[0] + R.hi[0]) / 2, jm = (R.lo[1] + R.hi[1]) / 2, km = (R.lo[2] + R.hi[2]) / 2;
        double nx, ny, nz;
        bc_normal(B, lin(B, im, jm, km), R.s_nd, nx, ny, nz);
        for (int l = 0; l < NG; ++l) {
          const int dist = l + 1;
          const long long ig = idx0 + dist * out, ii = idx0 - dist * out;
          const double rho = PR(0, ii), u = PR(1, ii), v = PR(2, ii), w = PR(3, ii), p = PR(4, ii);
          const double v_dot_n = u * nx + v * ny + w * nz;
          PR(0, ig) = rho;
          PR(1, ig) = u - 2.0 * v_dot_n * nx;
          PR(2, ig) = v - 2.0 * v_dot_n * ny;
          PR(3, ig) = w - 2.0 * v_dot_n * nz;
          PR(4, ig) = p;
          PR(5, ig) = PR(5, ii);
        }
      }
      if (P.method == 1) dif_average(B, idx0, out);
      break;
    }
    case 4: {
      // apply_farfield_bc (PhysicalBC.cpp:369-472)
      const double gama = P.gamma, gm1 = gama - 1.0;
      const double rho_inf = P.roo, u_inf = P.uoo, v_inf = P.voo, w_inf = P.woo, p_inf = P.poo;
      const double c_inf = sqrt(gama * p_inf / rho_inf);
      double nx, ny, nz;
      bc_normal(B, idx0, R.s_nd, nx, ny, nz);
      if (R.lr == -1) {
        nx = -nx;
        ny = -ny;
        nz = -nz;
      }
      const long long ii = idx0 - out;
      const double rho_in = PR(0, ii), u_in = PR(1, ii), v_in = PR(2, ii), w_in = PR(3, ii), p_in = PR(4, ii);
      const double c_in = sqrt(gama * p_in / rho_in);
      const double s_in = p_in / pow(rho_in, gama);
      const double s_inf = p_inf / pow(rho_inf, gama);
      const double vn_in = u_in * nx + v_in * ny + w_in * nz;
      const double vn_inf = u_inf * nx + v_inf * ny + w_inf * nz;
      const double vel_mag = sqrt(u_in * u_in + v_in * v_in + w_in * w_in);
      const double mach = vel_mag / c_in;
      double rho_b, u_b, v_b, w_b, p_b;
      if (mach < 1.0) {
        const double R_plus = vn_in + 2.0 * c_in / gm1;
        const double R_minus = vn_inf - 2.0 * c_inf / gm1;
        const double vn_b = 0.5 * (R_plus + R_minus);
        const double c_b = 0.25 * gm1 * (R_plus - R_minus);
        double s_b, u_ref, v_ref, w_ref, vn_ref;
        if (vn_b > 0.0) {
          s_b = s_in; u_ref = u_in; v_ref = v_in; w_ref = w_in; vn_ref = vn_in;
        } else {
          s_b = s_inf; u_ref = u_inf; v_ref = v_inf; w_ref = w_inf; vn_ref = vn_inf;
        }
        rho_b = pow(c_b * c_b / (gama * s_b), 1.0 / gm1);
        p_b = s_b * pow(rho_b, gama);
        u_b = u_ref + (vn_b - vn_ref) * nx;
        v_b = v_ref + (vn_b - vn_ref) * ny;
        w_b = w_ref + (vn_b - vn_ref) * nz;
      } else {
        if (vn_in > 0.0) {
          rho_b = rho_in; u_b = u_in; v_b = v_in; w_b = w_in; p_b = p_in;
        } else {
          rho_b = rho_inf; u_b = u_inf; v_b = v_inf; w_b = w_inf; p_b = p_inf;
        }
      }
      const double t_b = (mach * mach * gama) * p_b / rho_b;
      for (int l = 0; l < NG; ++l) {
        const int dist = l + 1;
        const long long ig = idx0 + dist * out;
        PR(0, ig) = (dist == 3) ? -rho_b : rho_b;
        PR(1, ig) = u_b;
        PR(2, ig) = v_b;
        PR(3, ig) = w_b;
        PR(4, ig) = p_b;
        PR(5, ig) = t_b;
      }
      break;
    }
    case 5: {
      // apply_freestream_bc (PhysicalBC.cpp:477-521)
      for (int l = 0; l < NG; ++l) {
        const long long ig = idx0 + (l + 1) * out;
        PR(0, ig) = P.roo;
        PR(1, ig) = P.uoo;
        PR(2, ig) = P.voo;
        PR(3, ig) = P.woo;
        PR(4, ig) = P.poo;
        PR(5, ig) = P.too;
      }
      break;
    }
    case 6: {
      // apply_extrapolation_bc (PhysicalBC.cpp:526-571)
      const long long is = idx0 - out;
      double v[6];
      for (int m = 0; m < 6; ++m) v[m] = PR(m, is);
      for (int l = 0; l < NG; ++l) {
        const long long ig = idx0 + (l + 1) * out;
        for (int m = 0; m < 6; ++m) PR(m, ig) = v[m];
      }
      break;
    }
    default:
      break;
  }
}

// ===========================================================================
// Derived state + dq := 0 (+ local time step when DO_DT)
// update_flow_states (src/solver/StateUpdater.cpp:15-168) and
// calculate_spectrum / calculate_local_dt_cell (src/solver/TimeIntegrator.cpp:20-125),
// one pass over the padded points.  The spectral radii are consumed in place
// (they are read nowhere else).  phydtime = min(1000, min dt*vol) via atomicMin
// on the bit pattern of a positive double.
// ===========================================================================
// calculate_spectrum + calculate_local_dt_cell (TimeIntegrator.cpp:20-125) from
// one point's values; km: its metrics.
template <typename S>
__device__ __forceinline__ S timestep_value(const ParamsDev& P, S rho, S u, S v, S w, S vol, S c, S mu, const S km[9]) {
  const S reynolds = (S)P.reynolds, csrv = (S)P.csrv;
  S sum_spec = S(0);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const S mx = km[3 * d], my = km[3 * d + 1], mz = km[3 * d + 2];
    const S U_contra = tabs(u * mx + v * my + w * mz);
    const S grad_len = tsqrt(mx * mx + my * my + mz * mz);
    const S spec = U_contra + c * grad_len;
    S specv = S(0);
    if (P.nvis == 1) {
      const S grad_sq = mx * mx + my * my + mz * mz;
      const S denom = reynolds * rho * vol + S(1.0e-30);
      specv = (S(2) * mu / denom) * grad_sq * csrv;
    }
    sum_spec += spec + specv;
  }
  const S dt_phys = (S)P.cfl / (sum_spec + S(1.0e-30));
  return dt_phys / vol;
}

// CTA-wide minimum written to part[blockIdx.x] (no same-address atomics: a
// few thousand of those serialize for milliseconds).
__device__ __forceinline__ void block_min_to(double v, double* part) {
  for (int off = 16; off > 0; off >>= 1) v = fmin(v, __shfl_down_sync(0xffffffffu, v, off));
  __shared__ double s_min[32];
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) s_min[w] = v;
  __syncthreads();
  if (w == 0) {
    const int nw = (blockDim.x + 31) >> 5;
    v = (l < nw) ? s_min[l] : 1000.0;
    for (int off = 16; off > 0; off >>= 1) v = fmin(v, __shfl_down_sync(0xffffffffu, v, off));
    if (l == 0) part[blockIdx.x] = v;
  }
}

// phydtime = min(1000, min over the partials) (TimeIntegrator.cpp:151-176), stored as bits.
__device__ __forceinline__ void dtmin_final_body(const double* __restrict__ part, int n,
                                                 unsigned long long* __restrict__ dtmin_bits);

static __global__ void __launch_bounds__(1024) k_dtmin_final(const double* __restrict__ part, int n,
                                                             unsigned long long* __restrict__ dtmin_bits) {
  dtmin_final_body(part, n, dtmin_bits);
}

__device__ __forceinline__ void dtmin_final_body(const double* __restrict__ part, int n,
                                                 unsigned long long* __restrict__ dtmin_bits) {
  double v = 1000.0;
  for (int t = threadIdx.x; t < n; t += 1024) v = fmin(v, part[t]);
  for (int off = 16; off > 0; off >>= 1) v = fmin(v, __shfl_down_sync(0xffffffffu, v, off));
  __shared__ double s_min[32];
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) s_min[w] = v;
  __syncthreads();
  if (w == 0) {
    v = s_min[l];
    for (int off = 16; off > 0; off >>= 1) v = fmin(v, __shfl_down_sync(0xffffffffu, v, off));
    if (l == 0) *dtmin_bits = (unsigned long long)__double_as_longlong(v);
  }
}

// CTAs per SM (256 threads each) the sweep-preparation kernels are compiled for
// (register cap 65536 / (256 n)), per precision: 385x257x129 in 64 blocks,
// k_tile_prep in FP32 0.62 ms at five, 0.573 at six, 0.560 at seven; in FP64
// 1.23 at three, 1.106 at four, 1.24 at five.
#ifndef ORION_PTWISE_MINB_F32
#define ORION_PTWISE_MINB_F32 6
#endif
#ifndef ORION_PTWISE_MINB_F64
#define ORION_PTWISE_MINB_F64 4
#endif
#ifndef ORION_STATE_MINB
#define ORION_STATE_MINB 4
#endif
template <typename T> struct PointwiseMinBlocks;
template <> struct PointwiseMinBlocks<float> { static constexpr int n = ORION_PTWISE_MINB_F32; };
template <> struct PointwiseMinBlocks<double> { static constexpr int n = ORION_PTWISE_MINB_F64; };

// One point a thread, every value it needs asked for before the first is used:
// what bounds it is the latency of its loads, and stores in between held the
// later ones back (385x257x129 mixed 0.83 -> 0.57 ms, plain 1.06 -> 0.72; at four
// CTAs an SM, three 0.57 and 0.74, five 0.52 and 0.82).  Arithmetic in the
// storage precision S of c, mu, dt (FP64 on the plain path).
template <typename S, bool DO_Q, bool DO_DT>
__global__ void __launch_bounds__(256, ORION_STATE_MINB) k_state(const BlockDev<S>* __restrict__ blocks, const Chunk* __restrict__ chunks,
                        double* __restrict__ dt_part) {
  const Chunk ch = chunks[blockIdx.x];
  const BlockDev<S>& B = blocks[ch.block];
  const ParamsDev& P = B.prm;
  double local_min = 1000.0;
  if ((int)threadIdx.x < ch.count) {
    const long long np = B.npad;
    const int nx = B.nx, ny = B.ny;
    const int i32 = (int)ch.start + threadIdx.x;  // padded index < 2^31
    const long long idx = i32;
    const int r32 = i32 / nx, i = i32 - r32 * nx;
    const int k = r32 / ny, j = r32 - k * ny;
    const bool inI = (i >= NG && i < NG + B.ni), inJ = (j >= NG && j < NG + B.nj), inK = (k >= NG && k < NG + B.nk);
    const int nin = (int)inI + (int)inJ + (int)inK;  // 3: interior, 2: ghost face slab
    double* const prim = B.prim;
    double pr[6];
#pragma unroll
    for (int m = 0; m < 6; ++m) pr[m] = prim[m * np + idx];
    S km[9], vol = S(0);
    double vol64 = 0.0;
    if (DO_DT && nin == 3) {
      const S* const met = FluxSrc<S>::metrics(B);
#pragma unroll
      for (int m = 0; m < 9; ++m) km[m] = met[m * np + idx];
      vol = FluxSrc<S>::vol(B)[idx];
      vol64 = B.vol[idx];
    }
    const int nvis = P.nvis;
    const S moo = (S)P.moo, visc = (S)P.visc;
    S T = (S)pr[5], cval = S(0), muv = S(0);
    if (nin >= 2) {  // update_thermodynamics_block
      S rho = (S)pr[0];
      if (nin == 2) rho = tabs(rho);
      const S a2 = (S)P.gamma * (S)pr[4] / rho;
      cval = tsqrt(tabs(a2));
      if (nvis == 1) T = (moo * moo) * a2;
    }
    if (nvis == 1) {  // update_viscosity_block (StateUpdater.cpp:75-92): whole padded array
      S tm = T;
      if (tm < S(1e-6)) tm = S(1e-6);
      muv = tm * tsqrt(tm) * (S(1) + visc) / (tm + visc);
      B.mu[idx] = muv;
    }
    if (nin >= 2) {
      B.c[idx] = cval;
      if (nvis == 1) prim[5 * np + idx] = (double)T;
      if (DO_Q) {  // update_conservative_block (StateUpdater.cpp:94-149), FP64
        const bool use_abs = (nin == 2);
        const double rc = (use_abs || pr[0] < 0.0) ? fabs(pr[0]) : pr[0];
        const double gm1_inv = 1.0 / (P.gamma - 1.0);
        B.q[idx] = rc;
        B.q[np + idx] = rc * pr[1];
        B.q[2 * np + idx] = rc * pr[2];
        B.q[3 * np + idx] = rc * pr[3];
        const double ke = 0.5 * rc * (pr[1] * pr[1] + pr[2] * pr[2] + pr[3] * pr[3]);
        B.q[4 * np + idx] = pr[4] * gm1_inv + ke;
      }
    }
#pragma unroll
    for (int m = 0; m < 5; ++m) B.dq[m * np + idx] = (S)0;
    if constexpr (sizeof(S) == 4) {  // the flux kernels' FP32 copy of prim, after the BCs and T
#pragma unroll
      for (int m = 0; m < 5; ++m) B.prim_f[m * np + idx] = (float)pr[m];
      B.prim_f[5 * np + idx] = (nin >= 2 && nvis == 1) ? (float)T : (float)pr[5];
    }
    if (DO_DT && nin == 3) {
      const S dtv = timestep_value<S>(P, (S)pr[0], (S)pr[1], (S)pr[2], (S)pr[3], vol, cval, muv, km);
      B.dt[idx] = dtv;
      const double dt_phys = (double)dtv * vol64;
      if (dt_phys < local_min) local_min = dt_phys;
    }
  }
  if (DO_DT) block_min_to(local_min, dt_part);
}

// time step alone (per-stage entry point): interior points of interior chunks
template <typename S>
__global__ void k_timestep(const BlockDev<S>* __restrict__ blocks, const Chunk* __restrict__ chunks,
                        double* __restrict__ dt_part) {
  const Chunk ch = chunks[blockIdx.x];
  const BlockDev<S> B = blocks[ch.block];
  const ParamsDev& P = B.prm;
  double local_min = 1000.0;
  for (int t = threadIdx.x; t < ch.count; t += blockDim.x) {
    const long long n = ch.start + t;  // interior index
    const int n32 = (int)n, r32 = n32 / B.ni;
    const int ii = n32 - r32 * B.ni, jj = r32 % B.nj, kk = r32 / B.nj;
    const long long idx = lin(B, NG + ii, NG + jj, NG + kk);
    const long long np = B.npad;
    S km[9];
    for (int m = 0; m < 9; ++m) km[m] = (S)__ldg(FluxSrc<S>::metrics(B) + m * np + idx);
    const S dtv = timestep_value<S>(P, (S)B.prim[idx], (S)B.prim[np + idx], (S)B.prim[2 * np + idx],
                                    (S)B.prim[3 * np + idx], FluxSrc<S>::vol(B)[idx], B.c[idx], B.mu[idx], km);
    B.dt[idx] = dtv;
    const double dt_phys = (double)dtv * B.vol[idx];
    if (dt_phys < local_min) local_min = dt_phys;
  }
  block_min_to(local_min, dt_part);
}


// ===========================================================================
// Node derivatives of (u,v,w,T) along xi, eta, zeta at interior points
// (compute_derivatives_cell + compute_node_deriv_line,
// src/solver/FluxComputer.cpp:13-67, 301-376).
// ===========================================================================
template <typename S, typename T>
__global__ void k_node_derivs(const BlockDev<S>* __restrict__ blocks, const Chunk* __restrict__ chunks) {
  const Chunk ch = chunks[blockIdx.x];
  const BlockDev<S>& B = blocks[ch.block];
  if ((int)threadIdx.x >= ch.count) return;
  const long long np = B.npad;
  const int n32 = (int)ch.start + threadIdx.x, r32 = n32 / B.ni;
  const int kk = r32 / B.nj, jj = r32 - kk * B.nj, ii = n32 - r32 * B.ni;
  const long long idx = lin(B, NG + ii, NG + jj, NG + kk);
  const S* const prim = FluxSrc<S>::prim(B) + idx;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int t = d == 0 ? ii : (d == 1 ? jj : kk), L = dim_along(B, d);
    const int st = (int)stride_along(B, d);  // padded indices are below 2^31
    // one-sided at the two points of a flagged end (ghost-3 density below zero)
    bool low = t <= 1, high = t >= L - 2;
    if (low) low = B.prim[idx - (long long)(t + NG) * st] < 0.0;
    if (high) high = B.prim[idx + (long long)(L + 2 - t) * st] < 0.0;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const S* const q = prim + (m < 3 ? m + 1 : 5) * np;
      T v;
      if (low || high) {
        const int in = low ? st : -st, far = low ? t : L - 1 - t;  // points from the end
        const S* const e = q - far * in;
        const T q1 = (T)e[0], q2 = (T)e[in], q3 = (T)e[2 * in], q4 = (T)e[3 * in];
        if (far == 0) v = div6(T(-11) * q1 + T(18) * q2 - T(9) * q3 + T(2) * q4);
        else v = div12(T(-3) * q1 + T(-10) * q2 + T(18) * q3 + T(-6) * q4 + T(1) * (T)e[4 * in]);
        if (!low) v = -v;
      } else {
        v = div12(T(8) * ((T)q[st] - (T)q[-st]) + T(-1) * ((T)q[2 * st] - (T)q[-2 * st]));
      }
      B.duvwt[(m + 4 * d) * np + idx] = (S)v;
    }
  }
}

// Register caps of the line kernels, as CTAs per SM of 256 threads (65536/(256*n)),
// per compute precision, measured on 385x257x129 in 64 blocks, the three
// directions: viscous FP32 four (2.45 ms; three 2.49, five 2.54), where its
// shared memory lets three CTAs be resident; FP64 two (4.55 ms without spills;
// three 5.68); inviscid FP32 four, FP64 three, as many as are resident
// (inviscid.cuh).
#ifndef ORION_VISC_MINB_F32
#define ORION_VISC_MINB_F32 4
#endif
#ifndef ORION_INV_MINB_F32
#define ORION_INV_MINB_F32 4
#endif
#ifndef ORION_VISC_MINB_F64
#define ORION_VISC_MINB_F64 2
#endif
#ifndef ORION_INV_MINB_F64
#define ORION_INV_MINB_F64 3
#endif
template <typename T> struct LineMinBlocks;
template <> struct LineMinBlocks<float> { static constexpr int visc = ORION_VISC_MINB_F32, inv = ORION_INV_MINB_F32; };
template <> struct LineMinBlocks<double> { static constexpr int visc = ORION_VISC_MINB_F64, inv = ORION_INV_MINB_F64; };

// ===========================================================================
// Interface residual averaging (HaloExchanger::average_interface_residuals,
// src/solver/HaloExchanger.cpp:186-398): pack dq/vol of every source window
// before any update, then each destination point applies its partners in
// region order: dq = 0.5 * (dens_t * vol + dq).
// ===========================================================================
template <typename S>
__global__ void k_iface_pack(const BlockDev<S>* __restrict__ blocks, const int* __restrict__ pk_block,
                             const long long* __restrict__ pk_idx, double* __restrict__ pack, int n) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const BlockDev<S> B = blocks[pk_block[t]];
  const long long idx = pk_idx[t];
  const double vol = B.vol[idx];
  for (int m = 0; m < 5; ++m) pack[(long long)t * 5 + m] = (double)B.dq[m * B.npad + idx] / vol;
}

template <typename S>
__global__ void k_iface_apply(const BlockDev<S>* __restrict__ blocks, const int* __restrict__ ap_block,
                              const long long* __restrict__ ap_idx, const int* __restrict__ ap_off,
                              const int* __restrict__ ap_slot, const double* __restrict__ pack, int n) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const BlockDev<S> B = blocks[ap_block[t]];
  const long long idx = ap_idx[t];
  const double vol_s = B.vol[idx];
  double q[5];
  for (int m = 0; m < 5; ++m) q[m] = (double)B.dq[m * B.npad + idx];
  for (int e = ap_off[t]; e < ap_off[t + 1]; ++e) {
    const long long sl = ap_slot[e];
    for (int m = 0; m < 5; ++m) {
      const double dens_t = pack[sl * 5 + m];
      q[m] = (double)(S)(0.5 * (dens_t * vol_s + q[m]));
    }
  }
  for (int m = 0; m < 5; ++m) B.dq[m * B.npad + idx] = (S)q[m];
}

// ===========================================================================
// LU-SGS / symmetric Gauss-Seidel (StateUpdater::update_solution,
// src/solver/StateUpdater.cpp:267-580) on the plane-major layout.
// Any order that visits a point after its lower face neighbours and before its
// upper ones reproduces the lexicographic sweeps exactly; the hyperplane order
// does, and each hyperplane is a contiguous, coalesced range here.
// ===========================================================================
__device__ __forceinline__ double sqrt_s(double x) { return sqrt(x); }
__device__ __forceinline__ float sqrt_s(float x) { return sqrtf(x); }

// Static skewed operands (metrics, vol, unit normals): refreshed whenever they are uploaded.
// FP32 shadows of one block's metrics and vol (padded, ghosts included).
static __global__ void k_metric_shadow(const BlockDev<float>* __restrict__ blocks, int b) {
  const BlockDev<float>& B = blocks[b];
  const long long np = B.npad;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < np; idx += (long long)gridDim.x * blockDim.x) {
    for (int m = 0; m < 9; ++m) B.met_f[m * np + idx] = (float)B.metrics[m * np + idx];
    B.vol_f[idx] = (float)B.vol[idx];
  }
}

// FP32 shadow of one block's prim (after an upload or the initial state).
static __global__ void k_prim_shadow(const BlockDev<float>* __restrict__ blocks, int b) {
  const BlockDev<float>& B = blocks[b];
  const long long np = B.npad;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < np; idx += (long long)gridDim.x * blockDim.x)
    for (int m = 0; m < 6; ++m) B.prim_f[m * np + idx] = (float)B.prim[m * np + idx];
}

template <typename S>
__global__ void k_skew_static(const BlockDev<S>* __restrict__ blocks, int b) {
  const BlockDev<S> B = blocks[b];
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < B.ncomp; c += (long long)gridDim.x * blockDim.x) {
    const int nat = B.sk_nat[c];
    for (int m = 0; m < 9; ++m) B.sk_metrics[m * B.ncomp + c] = (S)B.metrics[m * B.npad + nat];
    B.sk_vol[c] = (S)B.vol[nat];
    // unit normals of compute_flux_splitting (StateUpdater.cpp:231-249), per direction
    for (int d = 0; d < 3; ++d) {
      const S nx = B.sk_metrics[(3 * d) * B.ncomp + c], ny = B.sk_metrics[(3 * d + 1) * B.ncomp + c],
              nz = B.sk_metrics[(3 * d + 2) * B.ncomp + c];
      S grad_mag = sqrt_s(nx * nx + ny * ny + nz * nz);
      if (grad_mag < S(1.0e-30)) grad_mag = S(1.0e-30);
      const S inv_mag = S(1) / grad_mag;
      B.sk_nrm[(3 * d) * B.ncomp + c] = nx * inv_mag;
      B.sk_nrm[(3 * d + 1) * B.ncomp + c] = ny * inv_mag;
      B.sk_nrm[(3 * d + 2) * B.ncomp + c] = nz * inv_mag;
    }
  }
}

// What the sweeps need of one point besides its RHS: the diagonal coefficient
// 1/(1/dt + sum of radii) (get_diag_coeff, StateUpdater.cpp:267-295), the same
// in all four sweeps, and its quantities as a neighbour in
// compute_flux_splitting (:217-253) and visc_spectral_radius (:194-207).
template <typename T>
struct PrepPoint {
  T coed, H, c2, af, c, vcoef;
  __device__ __forceinline__ void form(const ParamsDev& P, T rho, T u, T v, T w, T p, const T km[9], T mu, T vol, T dt) {
    const T gamma = T(P.gamma), reynolds = T(P.reynolds);
    const T ra = spectral_radius<T>(rho, u, v, w, p, gamma, km[0], km[1], km[2]);
    const T rb = spectral_radius<T>(rho, u, v, w, p, gamma, km[3], km[4], km[5]);
    const T rc = spectral_radius<T>(rho, u, v, w, p, gamma, km[6], km[7], km[8]);
    T rva = T(0), rvb = T(0), rvc = T(0);
    vcoef = T(0);
    T rm = rho, pm = p;
    if (rm < T(1e-30)) rm = T(1e-30);
    if (pm < T(1e-30)) pm = T(1e-30);
    if (P.nvis == 1) {
      if (vol < T(1e-30)) vol = T(1e-30);
      const T rm_vol = rm * vol;
      vcoef = T(2) * mu / (tabs(reynolds) * rm_vol + T(1.0e-30));
      rva = visc_spectral_radius<T>(rho, mu, vol, reynolds, km[0], km[1], km[2]);
      rvb = visc_spectral_radius<T>(rho, mu, vol, reynolds, km[3], km[4], km[5]);
      rvc = visc_spectral_radius<T>(rho, mu, vol, reynolds, km[6], km[7], km[8]);
    }
    const T rad_sum = ra + rb + rc + rva + rvb + rvc;
    const T term = (T(1) / dt) + rad_sum;
    coed = T(1) / term;
    const T v2 = u * u + v * v + w * w;
    c2 = gamma * pm / rm;
    H = (gamma / (gamma - T(1))) * (pm / rm) + T(0.5) * v2;
    af = T(0.5) * (gamma - T(1)) * v2;
    c = tsqrt(c2);
  }
};

// Prep of the plane-major forms: gather prim, mu into the skewed layout; rhs =
// dq with physical-BC windows zeroed (set_boundary_dq_zero + the AoS copy,
// StateUpdater.cpp:447-570).
template <typename S, typename T>
__global__ void __launch_bounds__(256, PointwiseMinBlocks<T>::n) k_lusgs_prep(const BlockDev<S>* __restrict__ blocks, const Chunk* __restrict__ chunks) {
  const Chunk ch = chunks[blockIdx.x];
  const BlockDev<S> B = blocks[ch.block];
  const ParamsDev& P = B.prm;
  const long long np = B.npad, nc = B.ncomp;
  for (int t = threadIdx.x; t < ch.count; t += blockDim.x) {
    const long long c = ch.start + t;
    const int nat = B.sk_nat[c];
    const bool masked = B.bcmask[nat] != 0;
    for (int m = 0; m < 5; ++m) B.sk_rhs[m * nc + c] = masked ? (S)0 : B.dq[m * np + nat];
    const S* pr = FluxSrc<S>::prim(B);
    const T rho = (T)pr[nat], u = (T)pr[np + nat], v = (T)pr[2 * np + nat], w = (T)pr[3 * np + nat],
            p = (T)pr[4 * np + nat];
    B.sk_prim[c] = (S)rho;  // the operands of k_sweep_pairs
    B.sk_prim[nc + c] = (S)u;
    B.sk_prim[2 * nc + c] = (S)v;
    B.sk_prim[3 * nc + c] = (S)w;
    B.sk_prim[4 * nc + c] = (S)p;
    T km[9];
    for (int m = 0; m < 9; ++m) km[m] = (T)B.sk_metrics[m * nc + c];
    const T mu = (T)B.mu[nat];
    B.sk_mu[c] = (S)mu;
    PrepPoint<T> q;
    q.form(P, rho, u, v, w, p, km, mu, (T)B.sk_vol[c], (T)B.dt[nat]);
    B.sk_coed[c] = (S)q.coed;
    B.sk_nbq[c] = (S)u;
    B.sk_nbq[nc + c] = (S)v;
    B.sk_nbq[2 * nc + c] = (S)w;
    B.sk_nbq[3 * nc + c] = (S)q.H;
    B.sk_nbq[4 * nc + c] = (S)q.c2;
    B.sk_nbq[5 * nc + c] = (S)q.af;
  }
}

// Per face neighbour q of every point: the increment-independent coefficients of
// add_nb / add_nb_contrib (StateUpdater.cpp:326-343, 401-421): spectral radius of
// the neighbour with the point's metric, split eigenvalues l1 (and l4, l5 through
// x1, x2), ct_n, and half the viscous radius.  q = 0..2 lower i,j,k (sign +1),
// q = 3..5 upper (sign -1).
template <typename S, typename T>
__global__ void k_sweep_pairs(const BlockDev<S>* __restrict__ blocks, const Chunk* __restrict__ chunks) {
  const Chunk ch = chunks[blockIdx.x];
  const BlockDev<S> B = blocks[ch.block];
  const ParamsDev& P = B.prm;
  const long long nc = B.ncomp;
  const T gamma = T(P.gamma);
  for (int t = threadIdx.x; t < ch.count; t += blockDim.x) {
    const long long c = ch.start + t;
    int nb[6];
    for (int q = 0; q < 6; ++q) nb[q] = B.sk_nb[q * nc + c];
    for (int q = 0; q < 6; ++q) {
      if (nb[q] < 0) continue;
      const long long n = nb[q];
      const int d = q % 3;
      const T nx = (T)B.sk_metrics[(3 * d) * nc + c], ny = (T)B.sk_metrics[(3 * d + 1) * nc + c],
              nz = (T)B.sk_metrics[(3 * d + 2) * nc + c];
      const T rho = (T)B.sk_prim[n], um = (T)B.sk_prim[nc + n], vm = (T)B.sk_prim[2 * nc + n],
              wm = (T)B.sk_prim[3 * nc + n], p = (T)B.sk_prim[4 * nc + n];
      const T r = spectral_radius<T>(rho, um, vm, wm, p, gamma, nx, ny, nz);
      const T sign = q < 3 ? T(1) : T(-1);
      // compute_flux_splitting up to the increment-dependent part
      T rm = rho, pm = p;
      if (rm < T(1e-30)) rm = T(1e-30);
      if (pm < T(1e-30)) pm = T(1e-30);
      const T c2 = gamma * pm / rm;
      const T cm = tsqrt(c2);
      const T ct = nx * um + ny * vm + nz * wm + T(0);
      T grad_mag = tsqrt(nx * nx + ny * ny + nz * nz);
      if (grad_mag < T(1.0e-30)) grad_mag = T(1.0e-30);
      T l1 = ct;
      T l4 = ct + cm * grad_mag;
      T l5 = ct - cm * grad_mag;
      l1 = T(0.5) * (l1 + sign * r);
      l4 = T(0.5) * (l4 + sign * r);
      l5 = T(0.5) * (l5 + sign * r);
      const T x1 = (T(2) * l1 - l4 - l5) / (T(2) * c2);
      const T x2 = (l4 - l5) / (T(2) * cm);
      const T inv_mag = T(1) / grad_mag;
      const T ct_n = (ct - T(0)) * inv_mag;
      T rvh = T(0);
      if (P.nvis == 1) {
        T vol_nb = (T)B.sk_vol[n];
        if (vol_nb < T(1e-30)) vol_nb = T(1e-30);
        const T rv = visc_spectral_radius<T>(rho, (T)B.sk_mu[n], vol_nb, T(P.reynolds), nx, ny, nz);
        rvh = T(0.5) * rv;
      }
      S* out = B.sk_pair + (long long)(5 * q) * nc + c;
      out[0] = (S)l1;
      out[nc] = (S)x1;
      out[2 * nc] = (S)x2;
      out[3 * nc] = (S)ct_n;
      out[4 * nc] = (S)rvh;
    }
  }
}

enum SweepMode { SW_LUSGS_FWD = 0, SW_LUSGS_BWD = 1, SW_GS = 2 };

// The cooperative-grid form (ORION_SWEEP_GRID): all four sweeps in one
// persistent cooperative launch, software-pipelined.
// Every CTA walks the hyperplane sequence; for each hyperplane a thread owns at
// most one point of its CTA's first chunk (further chunks are handled in place).
// The point's operands that do not change during the sweep (metrics, diagonal
// coefficient, RHS or its own earlier increment, neighbour indices) are loaded
// before the grid barrier that ends the previous hyperplane, so after the
// barrier one round of independent L2 loads (the neighbours' state and fresh
// increments) precedes the arithmetic.  The barrier's wait is bounded: after
// spin_limit polls the kernel records an error and every CTA returns (the host
// reports ORION_E_TIMEOUT) instead of spinning forever.
struct SweepCtl {
  unsigned int counter;
  int error;   // a wait gave up: what the other waits look at
  int* host;   // the same in the host's memory, read there after the work has finished: no copy on any path
};

// err: a SweepCtl's error word.  A call, off the waits' code: inlined three
// times it made an FP64 sweep step 0.3% longer (97x49x33: 1.0043 -> 1.0073 ms).
static __device__ __noinline__ void sweep_gave_up(int* err) {
  atomicExch(err, 1);
  SweepCtl* const ctl = reinterpret_cast<SweepCtl*>(reinterpret_cast<char*>(err) - offsetof(SweepCtl, error));
  *(volatile int*)ctl->host = 1;
  __threadfence_system();
}

__device__ __forceinline__ bool grid_barrier(SweepCtl* ctl, unsigned int target, long long spin_limit) {
  __syncthreads();
  __shared__ int s_abort;
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(&ctl->counter, 1u);
    long long it = 0;
    int abort = 0;
    while (true) {
      const unsigned int v = *(volatile unsigned int*)&ctl->counter;
      if (v >= target) break;
      if (*(volatile int*)&ctl->error) { abort = 1; break; }
      if (++it > spin_limit) {
        sweep_gave_up(&ctl->error);
        abort = 1;
        break;
      }
      __nanosleep(32);
    }
    __threadfence();
    s_abort = abort;
  }
  __syncthreads();
  return s_abort == 0;
}

template <typename T>
struct SweepOps {
  int block;     // -1: no point
  int c;         // compact index
  int nb[6];     // neighbour compact indices: lower i,j,k then upper i,j,k; -1 outside the interior
  T coed;
  T own[5];      // -rhs (forward LU-SGS, GS) or the point's forward increment (backward LU-SGS)
};

template <typename S, typename T, int MODE>
__device__ __forceinline__ void sweep_fetch(const BlockDev<S>& B, int block, int c, SweepOps<T>& o) {
  const long long nc = B.ncomp;
  o.block = block;
  o.c = c;
  for (int q = 0; q < 6; ++q) {
    const bool used = (q < 3) ? (MODE == SW_LUSGS_FWD || MODE == SW_GS) : (MODE == SW_LUSGS_BWD || MODE == SW_GS);
    o.nb[q] = used ? B.sk_nb[q * nc + c] : -1;
  }
  o.coed = (T)B.sk_coed[c];
  for (int m = 0; m < 5; ++m) {
    if (MODE == SW_LUSGS_BWD) o.own[m] = (T)__ldcg(B.sk_dq + m * nc + c);
    else o.own[m] = -(T)B.sk_rhs[m * nc + c];
  }
}

// The increment-dependent part of add_nb / add_nb_contrib for neighbour q
// (compute_flux_splitting from dc on, StateUpdater.cpp:255-264, and the viscous
// off-diagonal term :334-343 / :410-421), accumulated into rhs0 in the
// reference's order.
// The increment-dependent arithmetic of one neighbour term, from its loaded
// operands (dn: neighbour increment; nq: u, v, w, H, c2, af of the neighbour;
// pc: l1, x1, x2, ct_n, rv/2 of the pair; nrm: the point's unit normal).
template <typename T, int MODE>
__device__ __forceinline__ void split_flux(int q, T gm1, int nvis, const T dn[5], const T nq[6], const T pc[5],
                                           const T nrm[3], T fs[5]) {
  const T drm = dn[0], dum = dn[1], dvm = dn[2], dwm = dn[3], dEm = dn[4];
  const T um = nq[0], vm = nq[1], wm = nq[2], H = nq[3], c2 = nq[4], af = nq[5];
  const T nx_n = nrm[0], ny_n = nrm[1], nz_n = nrm[2];
  const T l1 = pc[0], x1 = pc[1], x2 = pc[2], ct_n = pc[3], rvh = pc[4];
  const T dc = ct_n * drm - (nx_n * dum + ny_n * dvm + nz_n * dwm);
  const T dh = af * drm - gm1 * (um * dum + vm * dvm + wm * dwm - dEm);
  const T c2dc = c2 * dc;
  fs[0] = l1 * drm - dh * x1 - dc * x2;
  fs[1] = l1 * dum + (nx_n * c2dc - um * dh) * x1 + (nx_n * dh - um * dc) * x2;
  fs[2] = l1 * dvm + (ny_n * c2dc - vm * dh) * x1 + (ny_n * dh - vm * dc) * x2;
  fs[3] = l1 * dwm + (nz_n * c2dc - wm * dh) * x1 + (nz_n * dh - wm * dc) * x2;
  fs[4] = l1 * dEm + (ct_n * c2dc - H * dh) * x1 + (ct_n * dh - H * dc) * x2;
  const T sgn = q < 3 ? T(1) : T(-1);
  if (nvis == 1) {
    if (MODE == SW_GS) {
      for (int m = 0; m < 5; ++m) fs[m] += rvh * dn[m] * sgn;
    } else {
      for (int m = 0; m < 5; ++m) fs[m] += rvh * dn[m];
    }
  }
}

template <typename T, int MODE>
__device__ __forceinline__ void split_accumulate(int q, const T fs[5], T rhs0[5]) {
  if (MODE == SW_GS && q >= 3) {
    for (int m = 0; m < 5; ++m) rhs0[m] -= fs[m];
  } else {
    for (int m = 0; m < 5; ++m) rhs0[m] += fs[m];
  }
}

template <typename T, int MODE>
__device__ __forceinline__ void split_term(int q, T gm1, int nvis, const T dn[5], const T nq[6], const T pc[5],
                                           const T nrm[3], T rhs0[5]) {
  T fs[5];
  split_flux<T, MODE>(q, gm1, nvis, dn, nq, pc, nrm, fs);
  split_accumulate<T, MODE>(q, fs, rhs0);
}

template <typename S, typename T, int MODE>
__device__ __forceinline__ void sweep_term(const BlockDev<S>& B, T gm1, int nvis, const SweepOps<T>& o, int q,
                                           T rhs0[5]) {
  const long long nc = B.ncomp;
  const long long n = o.nb[q];
  const long long c = o.c;
  const int d = q % 3;
  T dn[5], nq[6], pc[5], nrm[3];
  for (int m = 0; m < 5; ++m) dn[m] = (T)__ldcg(B.sk_dq + m * nc + n);
  for (int k = 0; k < 6; ++k) nq[k] = (T)B.sk_nbq[k * nc + n];
  for (int k = 0; k < 3; ++k) nrm[k] = (T)B.sk_nrm[(3 * d + k) * nc + c];
  for (int k = 0; k < 5; ++k) pc[k] = (T)B.sk_pair[(5 * q + k) * nc + c];
  split_term<T, MODE>(q, gm1, nvis, dn, nq, pc, nrm, rhs0);
}

template <typename S, typename T, int MODE>
__device__ __forceinline__ void sweep_apply(const BlockDev<S>& B, const ParamsDev& P, const SweepOps<T>& o) {
  const long long nc = B.ncomp;
  const T gm1 = T(P.gamma) - T(1);
  T rhs0[5] = {T(0), T(0), T(0), T(0), T(0)};
  // lower neighbours first (i, j, k), then upper (i, j, k): the reference's order
  for (int q = 0; q < 6; ++q)
    if (o.nb[q] >= 0) sweep_term<S, T, MODE>(B, gm1, P.nvis, o, q, rhs0);
  for (int m = 0; m < 5; ++m) {
    S* d = B.sk_dq + m * nc + o.c;
    if (MODE == SW_LUSGS_FWD) *d = (S)((o.own[m] + rhs0[m]) * o.coed);
    else if (MODE == SW_LUSGS_BWD) *d = (S)(o.own[m] - rhs0[m] * o.coed);
    else *d = (S)((rhs0[m] + o.own[m]) * o.coed);
  }
}

// One hyperplane of one sweep for every block; chunks list contiguous compact ranges.
// Launched as a programmatic dependent of the previous hyperplane's launch:
// before griddepcontrol.wait it reads what no earlier hyperplane writes (the
// neighbour indices, the diagonal coefficient, the RHS) and prefetches its
// splitting coefficients into L2, so the launch and those DRAM reads overlap
// the previous hyperplane; after the wait (the previous grid has completed
// and its writes are visible) it reads the neighbours' increments.  It lets
// its own dependent launch only after its wait, so at most one hyperplane
// ahead is resident.
__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void grid_dep_launch() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p)); }

// Threads per SM the per-hyperplane kernel is compiled for (register cap
// 65536 / this): 512 measured fastest on the 64-block 385x257x129 case.
#ifndef ORION_SWEEP_SM_THREADS
#define ORION_SWEEP_SM_THREADS 512
#endif
template <typename S, typename T, int MODE, int NT>
__global__ void __launch_bounds__(NT, ORION_SWEEP_SM_THREADS / NT) k_sweep_plane(const BlockDev<S>* __restrict__ blocks,
                                                    const Chunk* __restrict__ chunks) {
  constexpr int Q0 = MODE == SW_LUSGS_BWD ? 3 : 0;
  constexpr int Q1 = MODE == SW_LUSGS_FWD ? 3 : 6;
  constexpr bool PRELOAD = sizeof(T) == 4;  // FP32: every static operand in registers before the wait
  const Chunk ch = chunks[blockIdx.x];
  const bool active = (int)threadIdx.x < ch.count;
  const BlockDev<S>& B = blocks[ch.block];
  // the case's parameters, from the block's own descriptor: loaded with its
  // other fields and used only after the wait.  Work before the wait beyond
  // issuing loads lengthens the chain: it competes with the previous
  // hyperplane's launch, which is still running on the same SMs (forming a GS
  // pass's stale-side terms there, or even gamma - 1, made the step slower).
  const double gamma_ld = B.prm.gamma;
  const int nvis = B.prm.nvis;
  const long long nc = B.ncomp;
  const int c = (int)ch.start + threadIdx.x;
  // pointers into registers now: griddepcontrol.wait clobbers memory, so
  // anything read through B after it would be reloaded from global memory
  S* const skdq = B.sk_dq;
  const S* const sknbq = B.sk_nbq;
  const S* const skpair = B.sk_pair;
  const S* const sknrm = B.sk_nrm;
  int nb[6];
  T coed = T(0), own[5];
  T nq[6][6], pc[6][5], nrm[3][3];
  if (active) {
#pragma unroll
    for (int q = Q0; q < Q1; ++q) nb[q] = B.sk_nb[q * nc + c];
    coed = (T)B.sk_coed[c];
    if (MODE != SW_LUSGS_BWD)
#pragma unroll
      for (int m = 0; m < 5; ++m) own[m] = -(T)B.sk_rhs[m * nc + c];
#pragma unroll
    for (int q = Q0; q < Q1; ++q) {
      if (nb[q] < 0) continue;
      if (PRELOAD) {
#pragma unroll
        for (int k = 0; k < 6; ++k) nq[q][k] = (T)B.sk_nbq[k * nc + nb[q]];
#pragma unroll
        for (int k = 0; k < 5; ++k) pc[q][k] = (T)B.sk_pair[(5 * q + k) * nc + c];
      } else {
        for (int k = 0; k < 5; ++k) prefetch_l2(B.sk_pair + (long long)(5 * q + k) * nc + c);
        for (int k = 0; k < 6; ++k) prefetch_l2(B.sk_nbq + (long long)k * nc + nb[q]);
      }
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      if (PRELOAD) {
#pragma unroll
        for (int k = 0; k < 3; ++k) nrm[d][k] = (T)B.sk_nrm[(3 * d + k) * nc + c];
      } else {
        for (int k = 0; k < 3; ++k) prefetch_l2(B.sk_nrm + (long long)(3 * d + k) * nc + c);
      }
    }
  }
  grid_dep_wait();
  grid_dep_launch();
  if (!active) return;
  if (MODE == SW_LUSGS_BWD)  // the forward increment: the launch just before may have written it
#pragma unroll
    for (int m = 0; m < 5; ++m) own[m] = (T)__ldcg(skdq + m * nc + c);
  // every neighbour increment in flight at once
  T dn[6][5];
#pragma unroll
  for (int q = Q0; q < Q1; ++q)
    if (nb[q] >= 0)
#pragma unroll
      for (int m = 0; m < 5; ++m) dn[q][m] = (T)__ldcg(skdq + m * nc + nb[q]);
  const T gm1 = T(gamma_ld) - T(1);
  T rhs0[5] = {T(0), T(0), T(0), T(0), T(0)};
  // lower neighbours first (i, j, k), then upper (i, j, k): the reference's order
#pragma unroll
  for (int q = Q0; q < Q1; ++q) {
    if (nb[q] < 0) continue;
    const int d = q % 3;
    if (!PRELOAD) {
      for (int k = 0; k < 6; ++k) nq[q][k] = (T)sknbq[k * nc + nb[q]];
      for (int k = 0; k < 5; ++k) pc[q][k] = (T)skpair[(5 * q + k) * nc + c];
      for (int k = 0; k < 3; ++k) nrm[d][k] = (T)sknrm[(3 * d + k) * nc + c];
    }
    split_term<T, MODE>(q, gm1, nvis, dn[q], nq[q], pc[q], nrm[d], rhs0);
  }
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    S* dst = skdq + m * nc + c;
    if (MODE == SW_LUSGS_FWD) *dst = (S)((own[m] + rhs0[m]) * coed);
    else if (MODE == SW_LUSGS_BWD) *dst = (S)(own[m] - rhs0[m] * coed);
    else *dst = (S)((rhs0[m] + own[m]) * coed);
  }
}

template <typename S, typename T, int MODE>
__device__ __forceinline__ bool persistent_pass(const BlockDev<S>* __restrict__ blocks, const Chunk* __restrict__ chunks,
                                                const int* __restrict__ off, int nlaunch, const ParamsDev& P,
                                                SweepCtl* ctl, unsigned int& target, long long spin_limit) {
  SweepOps<T> cur;
  cur.block = -1;
  // prefetch hyperplane 0
  {
    const int ci = off[0] + blockIdx.x;
    if (ci < off[1]) {
      const Chunk ch = chunks[ci];
      if ((int)threadIdx.x < ch.count)
        sweep_fetch<S, T, MODE>(blocks[ch.block], ch.block, (int)ch.start + threadIdx.x, cur);
    }
  }
  for (int t = 0; t < nlaunch; ++t) {
    if (cur.block >= 0) sweep_apply<S, T, MODE>(blocks[cur.block], P, cur);
    // further chunks of this hyperplane owned by this CTA (large hyperplanes only)
    for (int ci = off[t] + blockIdx.x + gridDim.x; ci < off[t + 1]; ci += gridDim.x) {
      const Chunk ch = chunks[ci];
      if ((int)threadIdx.x < ch.count) {
        SweepOps<T> x;
        sweep_fetch<S, T, MODE>(blocks[ch.block], ch.block, (int)ch.start + threadIdx.x, x);
        sweep_apply<S, T, MODE>(blocks[ch.block], P, x);
      }
    }
    // prefetch the next hyperplane's static operands, then wait for this one
    cur.block = -1;
    if (t + 1 < nlaunch) {
      const int ci = off[t + 1] + blockIdx.x;
      if (ci < off[t + 2]) {
        const Chunk ch = chunks[ci];
        if ((int)threadIdx.x < ch.count)
          sweep_fetch<S, T, MODE>(blocks[ch.block], ch.block, (int)ch.start + threadIdx.x, cur);
      }
    }
    target += gridDim.x;
    if (!grid_barrier(ctl, target, spin_limit)) return false;
  }
  return true;
}

template <typename S, typename T, int NT>
__global__ void __launch_bounds__(NT) k_sweeps_persistent(const BlockDev<S>* __restrict__ blocks,
                                                           const Chunk* __restrict__ fwd_chunks,
                                                           const int* __restrict__ fwd_off,
                                                           const Chunk* __restrict__ bwd_chunks,
                                                           const int* __restrict__ bwd_off, int nlaunch,
                                                           ParamsDev P, SweepCtl* ctl, long long spin_limit) {
  unsigned int target = 0;
  if (!persistent_pass<S, T, SW_LUSGS_FWD>(blocks, fwd_chunks, fwd_off, nlaunch, P, ctl, target, spin_limit)) return;
  if (!persistent_pass<S, T, SW_LUSGS_BWD>(blocks, bwd_chunks, bwd_off, nlaunch, P, ctl, target, spin_limit)) return;
  if (!persistent_pass<S, T, SW_GS>(blocks, fwd_chunks, fwd_off, nlaunch, P, ctl, target, spin_limit)) return;
  persistent_pass<S, T, SW_GS>(blocks, bwd_chunks, bwd_off, nlaunch, P, ctl, target, spin_limit);
}

// Cluster form of the four sweeps.  Mesh blocks are independent, so only the
// CTAs that share a block have to agree on hyperplane boundaries: each thread
// block cluster owns a group of mesh blocks and walks the hyperplanes of that
// group, separating consecutive hyperplanes with the hardware cluster barrier
// (release/acquire at cluster scope).  No cluster waits on another, so clusters
// may also run one after another.  Software-pipelined like the persistent form.
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

// The fields of a block the sweeps touch, staged in shared memory so no
// hyperplane pays a global load for a pointer.
template <typename S>
struct SweepBlock {
  S* dq;
  const int* nb;
  const S* coed;
  const S* rhs;
  const S* nbq;
  const S* pair;
  const S* nrm;
  long long nc;
};

// A thread's share of one hyperplane: up to two chunks, staged per pass.
struct SweepSlot {
  int block;  // -1: none
  int start;
  int count;
};

// Static operands of point c: neighbour indices, diagonal coefficient and the
// RHS (or, backward, the forward increment) into registers; the splitting
// coefficients, neighbour states and normals prefetched to L2, so that after
// the barrier only the neighbours' fresh increments miss.
template <typename S, typename T, int MODE>
__device__ __forceinline__ void cl_fetch(const SweepBlock<S>& B, int block, int c, SweepOps<T>& o) {
  const long long nc = B.nc;
  o.block = block;
  o.c = c;
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    const bool used = (q < 3) ? (MODE == SW_LUSGS_FWD || MODE == SW_GS) : (MODE == SW_LUSGS_BWD || MODE == SW_GS);
    o.nb[q] = used ? __ldg(B.nb + q * nc + c) : -1;
  }
  o.coed = (T)B.coed[c];
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    if (MODE == SW_LUSGS_BWD) o.own[m] = (T)__ldcg(B.dq + m * nc + c);
    else o.own[m] = -(T)B.rhs[m * nc + c];
  }
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    if (o.nb[q] < 0) continue;
    for (int k = 0; k < 5; ++k) prefetch_l2(B.pair + (long long)(5 * q + k) * nc + c);
    for (int k = 0; k < 6; ++k) prefetch_l2(B.nbq + (long long)k * nc + o.nb[q]);
  }
  for (int k = 0; k < 9; ++k) prefetch_l2(B.nrm + (long long)k * nc + c);
}

// Every neighbour's increment in flight at once, then the terms in the
// reference's order (split_term: the same arithmetic as the other forms).
template <typename S, typename T, int MODE>
__device__ __forceinline__ void cl_apply(const SweepBlock<S>& B, T gm1, int nvis, const SweepOps<T>& o) {
  const long long nc = B.nc;
  const long long c = o.c;
  T dn[6][5];
#pragma unroll
  for (int q = 0; q < 6; ++q)
    if (o.nb[q] >= 0)
#pragma unroll
      for (int m = 0; m < 5; ++m) dn[q][m] = (T)__ldcg(B.dq + m * nc + o.nb[q]);
  T rhs0[5] = {T(0), T(0), T(0), T(0), T(0)};
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    if (o.nb[q] < 0) continue;
    const int d = q % 3;
    T nq[6], pc[5], nrm[3];
    for (int k = 0; k < 6; ++k) nq[k] = (T)B.nbq[k * nc + o.nb[q]];
    for (int k = 0; k < 5; ++k) pc[k] = (T)B.pair[(5 * q + k) * nc + c];
    for (int k = 0; k < 3; ++k) nrm[k] = (T)B.nrm[(3 * d + k) * nc + c];
    split_term<T, MODE>(q, gm1, nvis, dn[q], nq, pc, nrm, rhs0);
  }
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    S* d = B.dq + m * nc + c;
    if (MODE == SW_LUSGS_FWD) *d = (S)((o.own[m] + rhs0[m]) * o.coed);
    else if (MODE == SW_LUSGS_BWD) *d = (S)(o.own[m] - rhs0[m] * o.coed);
    else *d = (S)((rhs0[m] + o.own[m]) * o.coed);
  }
}

template <typename S, typename T, int MODE>
__device__ __forceinline__ void cluster_pass(const SweepBlock<S>* sb, const Chunk* __restrict__ chunks,
                                             const int* __restrict__ off, int nlaunch, int rank, int csize,
                                             const ParamsDev& P, SweepSlot* slots) {
  const T gm1 = T(P.gamma) - T(1);
  // stage this CTA's chunk of every hyperplane (two per hyperplane)
  __syncthreads();
  for (int x = threadIdx.x; x < 2 * nlaunch; x += blockDim.x) {
    const int t = x >> 1, r = x & 1;
    const int ci = off[t] + rank + r * csize;
    SweepSlot sl{-1, 0, 0};
    if (ci < off[t + 1]) {
      const Chunk ch = chunks[ci];
      sl = SweepSlot{ch.block, (int)ch.start, ch.count};
    }
    slots[x] = sl;
  }
  __syncthreads();
  SweepOps<T> cur[2];
  auto fetch = [&](int t) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const SweepSlot sl = slots[2 * t + r];
      cur[r].block = -1;
      if (sl.block >= 0 && (int)threadIdx.x < sl.count)
        cl_fetch<S, T, MODE>(sb[sl.block], sl.block, sl.start + threadIdx.x, cur[r]);
    }
  };
  fetch(0);
  for (int t = 0; t < nlaunch; ++t) {
#pragma unroll
    for (int r = 0; r < 2; ++r)
      if (cur[r].block >= 0) cl_apply<S, T, MODE>(sb[cur[r].block], gm1, P.nvis, cur[r]);
    // chunks beyond the two staged ones (very large hyperplanes only)
    for (int ci = off[t] + rank + 2 * csize; ci < off[t + 1]; ci += csize) {
      const Chunk ch = chunks[ci];
      if ((int)threadIdx.x < ch.count) {
        SweepOps<T> x;
        cl_fetch<S, T, MODE>(sb[ch.block], ch.block, (int)ch.start + threadIdx.x, x);
        cl_apply<S, T, MODE>(sb[ch.block], gm1, P.nvis, x);
      }
    }
    // publish this hyperplane, fetch the next one's static operands, then wait
    cluster_arrive();
    if (t + 1 < nlaunch) fetch(t + 1);
    cluster_wait();
  }
}

template <typename S, typename T, int NT>
__global__ void __launch_bounds__(NT, 1) k_sweeps_cluster(const BlockDev<S>* __restrict__ blocks, int nblocks,
                                                          const Chunk* __restrict__ fwd_chunks,
                                                          const int* __restrict__ fwd_off,
                                                          const Chunk* __restrict__ bwd_chunks,
                                                          const int* __restrict__ bwd_off,
                                                          const int* __restrict__ grp_base,
                                                          const int* __restrict__ grp_nplanes, ParamsDev P) {
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SweepBlock<S>* sb = reinterpret_cast<SweepBlock<S>*>(smem_raw);
  SweepSlot* slots = reinterpret_cast<SweepSlot*>(smem_raw + sizeof(SweepBlock<S>) * nblocks);
  for (int b = threadIdx.x; b < nblocks; b += blockDim.x) {
    const BlockDev<S>& B = blocks[b];
    sb[b] = SweepBlock<S>{B.sk_dq, B.sk_nb, B.sk_coed, B.sk_rhs, B.sk_nbq, B.sk_pair, B.sk_nrm, B.ncomp};
  }
  cg::cluster_group cl = cg::this_cluster();
  const int csize = (int)cl.num_blocks();
  const int rank = (int)cl.block_rank();
  const int g = blockIdx.x / csize;
  const int base = grp_base[g], n = grp_nplanes[g];
  cluster_pass<S, T, SW_LUSGS_FWD>(sb, fwd_chunks, fwd_off + base, n, rank, csize, P, slots);
  cluster_pass<S, T, SW_LUSGS_BWD>(sb, bwd_chunks, bwd_off + base, n, rank, csize, P, slots);
  cluster_pass<S, T, SW_GS>(sb, fwd_chunks, fwd_off + base, n, rank, csize, P, slots);
  cluster_pass<S, T, SW_GS>(sb, bwd_chunks, bwd_off + base, n, rank, csize, P, slots);
}

// Finish, per interior point in natural order: zero the physical-BC windows
// (set_boundary_dq_zero), bring the swept increment back to the natural
// layout, limited update (update_limited) and, when DO_RES, the residual
// partials (ResidualMonitor::compute).
template <typename S>
__device__ __forceinline__ void limited_update(const BlockDev<S>& B, const ParamsDev& P, long long idx,
                                               const double pr[5], const double dq[5]);
__device__ __forceinline__ void res_combine(double& sum, double& mx, long long& key, double osum, double omx,
                                            long long okey);
template <int NT>
__device__ __forceinline__ void block_reduce_res(double& sum, double& mx, long long& key);

// The finish kernel asks for every value before its first store (385x257x129
// mixed 0.67 -> 0.50 ms, plain 0.81 -> 0.66).
// CTAs per SM it is compiled for (register cap 65536 / (NT n)), 385x257x129:
// mixed 0.55 ms at three, 0.50 at four, 0.515 at five; plain 0.65, 0.65, 0.755.
#ifndef ORION_FINISH_MINB
#define ORION_FINISH_MINB 4
#endif
// Where interior point (ii, jj, kk) is in the block's tile arrays
// (sweep_tiles.cuh): slot of its wave's first line, its line, lines per wave.
struct TileSlot {
  long long wave;
  int line, nl;
  // its first piece in an array of `pieces` per point; pieces nl apart
  template <typename V>
  __device__ __forceinline__ V* run(char* base, int pieces) const {
    return reinterpret_cast<V*>(base) + wave * pieces + line;
  }
};
template <typename S>
__device__ __forceinline__ TileSlot tile_slot(const BlockDev<S>& B, int ii, int jj, int kk) {
  const int4 a = __ldg(B.t_j + jj), b = __ldg(B.t_k + kk);  // {tile column, line in it, width}, {tile row, ...}
  const int nl = a.z * b.z;
  return TileSlot{__ldg(B.t_base + b.x * B.tJ + a.x) + (long long)(ii + a.y + b.y) * nl, b.y * a.z + a.y, nl};
}
// The swept increment of a point.
__device__ __forceinline__ void tile_increment(const BlockDev<float>& B, const TileSlot& at, float d[5]) {
  const float4* const p = at.run<float4>(B.tl_nb, 3);
  const float4 a = __ldcs(p + 2 * at.nl);
  d[0] = a.x;
  d[1] = a.y;
  d[2] = a.z;
  d[3] = a.w;
  d[4] = __ldcs(reinterpret_cast<const float*>(p + at.nl) + 3);
}
__device__ __forceinline__ void tile_increment(const BlockDev<double>& B, const TileSlot& at, double d[5]) {
  const double2* const p = at.run<double2>(B.tl_nb, 8);
  const double2 a = __ldcs(p + 5 * at.nl), b = __ldcs(p + 6 * at.nl);
  d[0] = a.x;
  d[1] = a.y;
  d[2] = b.x;
  d[3] = b.y;
  d[4] = __ldcs(reinterpret_cast<const double*>(p + 7 * at.nl));
}

template <typename S, bool DO_RES, bool TILES, int NT>
__global__ void __launch_bounds__(NT, ORION_FINISH_MINB) k_sweep_finish(const BlockDev<S>* __restrict__ blocks,
                                                     const Chunk* __restrict__ chunks, ResPartial* __restrict__ partials) {
  // Natural order (interior index n = i + ni*(j + nj*k)): prim, dq, vol, dt
  // and the mask are read and written coalesced; only the swept increment is
  // gathered, from its tile slot or from the plane-major layout at
  // c = koff[s*nk + k] + (j - jlo(s,k)).
  const Chunk ch = chunks[blockIdx.x];
  const BlockDev<S> B = blocks[ch.block];
  const ParamsDev& P = B.prm;
  const long long np = B.npad, nc = B.ncomp;
  double sum = 0.0, mx = -1.0;
  long long key = (long long)0x7fffffffffffffffLL;
  if ((int)threadIdx.x < ch.count) {
    const long long n = ch.start + threadIdx.x;
    const int n32 = (int)n, r32 = n32 / B.ni;
    const int kk = r32 / B.nj, jj = r32 - kk * B.nj, ii = n32 - r32 * B.ni;
    const long long idx = lin(B, NG + ii, NG + jj, NG + kk);
    // every load before the first store
    double pr[5], vol = 0.0, dt = 0.0;
#pragma unroll
    for (int m = 0; m < 5; ++m) pr[m] = B.prim[m * np + idx];
    if (DO_RES) {
      vol = B.vol[idx];
      dt = (double)B.dt[idx];
    }
    const bool masked = B.bcmask[idx] != 0;
    S sw[5];
    if (TILES) {
      tile_increment(B, tile_slot(B, ii, jj, kk), sw);
    } else {
      const int sp = ii + jj + kk;
      const int jlo = sp - kk - (B.ni - 1) > 0 ? sp - kk - (B.ni - 1) : 0;
      const long long c = (long long)__ldg(B.koff + (long long)sp * B.nk + kk) + (jj - jlo);
      for (int m = 0; m < 5; ++m) sw[m] = __ldcs(B.sk_dq + m * nc + c);
    }
    double dq[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      const S v = masked ? (S)0 : sw[m];
      B.dq[m * np + idx] = v;
      dq[m] = (double)v;
    }
    limited_update(B, P, idx, pr, dq);
    if (DO_RES) {
      if (vol < 1e-30) vol = 1e-30;
      if (dt < 1e-30) dt = 1e-30;
      const double inv_factor = 1.0 / (dt * vol);
      const long long kbase = (B.int_base + n) * 5;
      for (int m = 0; m < 5; ++m) {
        const double res = fabs(dq[m]) * inv_factor;
        sum += res * res;
        if (res > mx || (res == mx && kbase + m < key)) {
          mx = res;
          key = kbase + m;
        }
      }
    }
  }
  if (DO_RES) {
    block_reduce_res<NT>(sum, mx, key);
    if (threadIdx.x == 0) partials[blockIdx.x] = ResPartial{sum, mx, key};
  }
}

// ===========================================================================
// update_limited (StateUpdater.cpp:447-542) and the residual
// (ResidualMonitor::compute, src/solver/ResidualMonitor.cpp:11-137): per-CTA
// partial sums and maxima with the lexicographic location key; a single CTA
// combines them in fixed order.
// ===========================================================================
template <typename S>
__device__ __forceinline__ void limited_update(const BlockDev<S>& B, const ParamsDev& P, long long idx,
                                               const double pr[5], const double dq[5]) {
  const long long np = B.npad;
  const double gm1 = P.gamma - 1.0;
  const double r = pr[0], u = pr[1], v = pr[2], w = pr[3], p = pr[4];
  const double E = p / gm1 + 0.5 * r * (u * u + v * v + w * w);
  double qn[5];
  qn[0] = r + dq[0];
  qn[1] = r * u + dq[1];
  qn[2] = r * v + dq[2];
  qn[3] = r * w + dq[3];
  qn[4] = E + dq[4];
  double r_n = qn[0];
  double inv_r = 1.0 / r_n;
  const double a = qn[1] * inv_r, b = qn[2] * inv_r, c = qn[3] * inv_r;
  const double p_n = gm1 * (qn[4] - 0.5 * r_n * (a * a + b * b + c * c));
  const double dp_p = fabs((p_n - p) / p);
  const double term = tmax(0.0, -0.3 + dp_p);
  const double Fa = 1.0 / (1.0 + 2.0 * term);
  double qf[5];
  qf[0] = r + dq[0] * Fa;
  qf[1] = r * u + dq[1] * Fa;
  qf[2] = r * v + dq[2] * Fa;
  qf[3] = r * w + dq[3] * Fa;
  qf[4] = E + dq[4] * Fa;
  r_n = qf[0];
  inv_r = 1.0 / r_n;
  const double u_n = qf[1] * inv_r, v_n = qf[2] * inv_r, w_n = qf[3] * inv_r;
  const double p_nf = gm1 * (qf[4] - 0.5 * r_n * (u_n * u_n + v_n * v_n + w_n * w_n));
  if (!(r_n <= 1e-6 || p_nf <= 1e-6)) {
    B.prim[idx] = r_n;
    B.prim[np + idx] = u_n;
    B.prim[2 * np + idx] = v_n;
    B.prim[3 * np + idx] = w_n;
    B.prim[4 * np + idx] = p_nf;
  }
}

__device__ __forceinline__ void res_combine(double& sum, double& mx, long long& key, double osum, double omx,
                                            long long okey) {
  sum += osum;
  if (omx > mx || (omx == mx && okey < key)) {
    mx = omx;
    key = okey;
  }
}

template <int NT>
__device__ __forceinline__ void block_reduce_res(double& sum, double& mx, long long& key) {
  // warp then CTA tree, fixed shape => deterministic
  for (int off = 16; off > 0; off >>= 1) {
    const double os = __shfl_down_sync(0xffffffffu, sum, off);
    const double om = __shfl_down_sync(0xffffffffu, mx, off);
    const long long ok = __shfl_down_sync(0xffffffffu, key, off);
    res_combine(sum, mx, key, os, om, ok);
  }
  __shared__ double s_sum[NT / 32];
  __shared__ double s_max[NT / 32];
  __shared__ long long s_key[NT / 32];
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) {
    s_sum[w] = sum;
    s_max[w] = mx;
    s_key[w] = key;
  }
  __syncthreads();
  if (w == 0) {
    sum = (l < NT / 32) ? s_sum[l] : 0.0;
    mx = (l < NT / 32) ? s_max[l] : -1.0;
    key = (l < NT / 32) ? s_key[l] : (long long)0x7fffffffffffffffLL;
    for (int off = 16; off > 0; off >>= 1) {
      const double os = __shfl_down_sync(0xffffffffu, sum, off);
      const double om = __shfl_down_sync(0xffffffffu, mx, off);
      const long long ok = __shfl_down_sync(0xffffffffu, key, off);
      res_combine(sum, mx, key, os, om, ok);
    }
  }
}

template <typename S, int NT>
__global__ void __launch_bounds__(NT) k_update_res(const BlockDev<S>* __restrict__ blocks, const Chunk* __restrict__ chunks,
                                                    ResPartial* __restrict__ partials) {
  const Chunk ch = chunks[blockIdx.x];
  const BlockDev<S> B = blocks[ch.block];
  const long long np = B.npad;
  double sum = 0.0, mx = -1.0;
  long long key = (long long)0x7fffffffffffffffLL;
  for (int t = threadIdx.x; t < ch.count; t += NT) {
    const long long n = ch.start + t;
    const int n32 = (int)n, r32 = n32 / B.ni;
    const int ii = n32 - r32 * B.ni, jj = r32 % B.nj, kk = r32 / B.nj;
    const long long idx = lin(B, NG + ii, NG + jj, NG + kk);
    double dq[5];
    for (int m = 0; m < 5; ++m) dq[m] = (double)B.dq[m * np + idx];
    double vol = B.vol[idx];
    double dt = (double)B.dt[idx];
    if (vol < 1e-30) vol = 1e-30;
    if (dt < 1e-30) dt = 1e-30;
    const double inv_factor = 1.0 / (dt * vol);
    const long long kbase = (B.int_base + n) * 5;
    for (int m = 0; m < 5; ++m) {
      const double res = fabs(dq[m]) * inv_factor;
      sum += res * res;
      if (res > mx || (res == mx && kbase + m < key)) {
        mx = res;
        key = kbase + m;
      }
    }
  }
  block_reduce_res<NT>(sum, mx, key);
  if (threadIdx.x == 0) partials[blockIdx.x] = ResPartial{sum, mx, key};
}

template <typename S>
__device__ __forceinline__ void res_final_body(const BlockDev<S>* __restrict__ blocks, int nblocks,
                                               const ResPartial* __restrict__ partials, int npart,
                                               long long total_points, const unsigned long long* dtmin_bits,
                                               ResidualOut* __restrict__ hist, int* __restrict__ counter,
                                               int capacity, ResPartial* __restrict__ total);

template <typename S>
__global__ void __launch_bounds__(1024) k_res_final(const BlockDev<S>* __restrict__ blocks, int nblocks,
                                                     const ResPartial* __restrict__ partials, int npart,
                                                     long long total_points, const unsigned long long* dtmin_bits,
                                                     ResidualOut* __restrict__ hist, int* __restrict__ counter,
                                                     int capacity, ResPartial* __restrict__ total) {
  res_final_body<S>(blocks, nblocks, partials, npart, total_points, dtmin_bits, hist, counter, capacity, total);
}

// One CTA per case of a group: that case's minimum time step (dt_part) or
// residual statistics (partials) over its own range, in the same order as
// the case's own launches, into the case's own result slots.
static __global__ void __launch_bounds__(1024) k_dtmin_group(const GroupMember* __restrict__ members,
                                                             const double* __restrict__ dt_part) {
  const GroupMember& m = members[blockIdx.x];
  dtmin_final_body(dt_part + m.pad_off, m.pad_n, m.dtmin);
}

template <typename S>
__global__ void __launch_bounds__(1024) k_res_final_group(const GroupMember* __restrict__ members,
                                                           const ResPartial* __restrict__ partials, int capacity) {
  const GroupMember& m = members[blockIdx.x];
  res_final_body<S>(static_cast<const BlockDev<S>*>(m.blocks), m.nblocks, partials + m.part_off, m.part_n,
                    m.total_points, m.dtmin, m.hist, m.counter, capacity, m.total);
}

template <typename S>
__device__ __forceinline__ void res_final_body(const BlockDev<S>* __restrict__ blocks, int nblocks,
                                               const ResPartial* __restrict__ partials, int npart,
                                               long long total_points, const unsigned long long* dtmin_bits,
                                               ResidualOut* __restrict__ hist, int* __restrict__ counter,
                                               int capacity, ResPartial* __restrict__ total) {
  double sum = 0.0, mx = -1.0;
  long long key = (long long)0x7fffffffffffffffLL;
  for (int t = threadIdx.x; t < npart; t += 1024) {
    const ResPartial p = partials[t];
    res_combine(sum, mx, key, p.sum, p.max, p.key);
  }
  block_reduce_res<1024>(sum, mx, key);
  if (threadIdx.x == 0) {
    if (total) *total = ResPartial{sum, mx, key};
    ResidualOut r;
    r.rms = total_points > 0 ? sqrt(sum / (double)total_points) : 0.0;
    r.max = mx;
    const long long pt = key / 5;
    int b = 0;
    for (int q = 0; q < nblocks; ++q) {
      const BlockDev<S>& B = blocks[q];
      if (pt >= B.int_base && pt < B.int_base + (long long)B.ni * B.nj * B.nk) b = q;
    }
    const BlockDev<S>& B = blocks[b];
    const long long n = pt - B.int_base;
    r.loc[0] = b;
    r.loc[1] = (int)(n % B.ni) + 1;
    r.loc[2] = (int)((n / B.ni) % B.nj) + 1;
    r.loc[3] = (int)(n / ((long long)B.ni * B.nj)) + 1;
    r.loc[4] = (int)(key % 5) + 1;
    r.pad = 0;
    r.phydtime = __longlong_as_double((long long)*dtmin_bits);
    const int c = *counter;
    hist[c % capacity] = r;
    *counter = c + 1;
  }
}

// ===========================================================================
// Initial flow on the device: freestream + splitmix64 noise + EOS temperature
// (initialize_flow / update_temperature, src/preprocess/InitialCondition.cpp:7-147).
// ===========================================================================
__device__ __forceinline__ double splitmix_uniform(unsigned long long seed, unsigned long long n) {
  unsigned long long z = seed + n * 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z = z ^ (z >> 31);
  return (double)(z >> 11) * (1.0 / 9007199254740992.0);
}

template <typename S>
__global__ void k_init_flow(const BlockDev<S>* __restrict__ blocks, const Chunk* __restrict__ chunks,
                            const long long* __restrict__ pad_base, unsigned long long seed, double amp) {
  const Chunk ch = chunks[blockIdx.x];
  const BlockDev<S> B = blocks[ch.block];
  const ParamsDev& P = B.prm;
  const long long np = B.npad;
  for (int t = threadIdx.x; t < ch.count; t += blockDim.x) {
    const long long idx = ch.start + t;
    const unsigned long long n = (unsigned long long)(pad_base[ch.block] + idx);
    double rho = P.roo, u = P.uoo;
    if (amp != 0.0) {
      const double r1 = splitmix_uniform(seed, 2 * n + 1);
      const double r2 = splitmix_uniform(seed, 2 * n + 2);
      rho = rho * (1.0 + amp * (2.0 * r1 - 1.0));
      u = u * (1.0 + amp * (2.0 * r2 - 1.0));
    }
    const double p = P.poo;
    B.prim[idx] = rho;
    B.prim[np + idx] = u;
    B.prim[2 * np + idx] = P.voo;
    B.prim[3 * np + idx] = P.woo;
    B.prim[4 * np + idx] = p;
    double T = P.too;
    if (P.nvis == 1) {
      double r = rho;
      if (r < 1.0e-30) r = 1.0e-30;
      const double a2 = P.gamma * p / r;
      T = (P.moo * P.moo) * a2;
    }
    B.prim[5 * np + idx] = T;
    B.q[idx] = P.roo;
    B.q[np + idx] = P.roo * P.uoo;
    B.q[2 * np + idx] = P.roo * P.voo;
    B.q[3 * np + idx] = P.roo * P.woo;
    const double v2 = P.uoo * P.uoo + P.voo * P.voo + P.woo * P.woo;
    B.q[4 * np + idx] = P.poo / (P.gamma - 1.0) + 0.5 * P.roo * v2;
    for (int m = 0; m < 5; ++m) B.dq[m * np + idx] = (S)0;
  }
}

}  // namespace orion
