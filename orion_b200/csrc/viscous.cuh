// Viscous RHS along one direction (compute_viscous_flux_block,
// src/solver/FluxComputer.cpp:466-722, with interp_line_to_half :129-178,
// compute_half_deriv_line :72-124, transform_derivs_to_phys :183-205,
// compute_viscous_flux_1d :210-252, compute_flux_diff_1d :257-296).
//
// A CTA takes NL neighbouring grid lines of one block and a chunk of points
// along them.  It stages the 23 values a face interpolates (velocity and
// temperature, viscosity, Jacobian, metrics, cross derivatives) once per point
// in shared memory, forms the faces' fluxes from them, and adds the 6th-order
// difference to dq (a face used to read 92 values from L1 and L2, each with a
// 64-bit address).  What bounds it: the phases' latency and shared-memory reads,
// 92 a face, with three (FP32) or two CTAs an SM: on 193x97x65 an instruction
// issues in 30-48% of the cycles (FP64 23-32%), the shared-memory pipe works in
// 33-56% and the FP64 pipe in 17-25%; the stalls are the barriers between the
// phases and the shared-memory queue.  The divisions by 24 and 1920 are products with the rounded
// reciprocal, corrected to the division's rounding (quotient).  385x257x129 in
// 64 blocks, the three directions: mixed 3.34 -> 2.45 ms, plain 6.19 -> 4.55;
// 97x49x33 mixed 0.146 -> 0.054 (chunks give small grids more CTAs).
#pragma once

#include "device_types.cuh"
#include "kernels.cuh"
#include "numerics.cuh"

namespace orion {

template <int D, typename T> struct ViscShape {
  static constexpr int NL = (D == 0 ? 4 : 8) * 8 / (int)sizeof(T);
  static constexpr int CM = D == 0 ? 64 : 32;
  static constexpr int NT = 256;
  static constexpr int NS = CM + 8;  // staged points
  static constexpr int NF = CM + 5;  // faces
  static constexpr int NV = 23;
  static constexpr size_t smem = sizeof(T) * NL * ((size_t)NV * NS + 4 * NF);
};

template <int D, typename S, typename T>
__global__ void __launch_bounds__(256, LineMinBlocks<T>::visc) k_viscous(const BlockDev<S>* __restrict__ blocks,
                                                                         const LineChunk* __restrict__ chunks) {
  using Z = ViscShape<D, T>;
  constexpr int NL = Z::NL, NS = Z::NS, NF = Z::NF;
  constexpr int QS = D == 0 ? 1 : NL;          // step along the line in shared memory
  constexpr int QN = NS * NL, FN = NF * NL;    // one staged variable, one flux component
  constexpr int VU = 0, VMU = 4, VVOL = 5, VMET = 6, VX = 15;
  constexpr int D1 = D == 0 ? 1 : 0, D2 = D == 2 ? 1 : 2;  // the other directions, ascending
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* const Q = reinterpret_cast<T*>(smem_raw);
  T* const F = Q + Z::NV * QN;
  __shared__ unsigned char s_flag[NL];
  __shared__ long long s_line[NL];
  const LineChunk ch = chunks[blockIdx.x];
  const BlockDev<S>& B = blocks[ch.block];
  const ParamsDev& P = B.prm;
  const long long np = B.npad;
  const int L = dim_along(B, D);
  const long long st = stride_along(B, D);
  const T cp = T(1) / ((T(P.gamma) - T(1)) * T(P.moo) * T(P.moo));
  const T cp_prl = cp / T(P.prl);
  const T re_inv = (fabs(P.reynolds) > 1.0e-30) ? T(1) / T(P.reynolds) : T(0);
  const int fA = max(0, ch.c0 - 2), fB = min(L, ch.c1 + 2);
  const int nf = fB - fA + 1, ns = nf + 3;  // staged from point fA - 2
  auto q_at = [&](int lane, int x) { return D == 0 ? lane * NS + x : x * NL + lane; };
  auto f_at = [&](int lane, int x) { return D == 0 ? lane * NF + x : x * NL + lane; };
  auto item = [&](int it, int n, int& lane, int& x) {
    if (D == 0) {
      lane = it / n;
      x = it - lane * n;
    } else {
      x = it / NL;
      lane = it - x * NL;
    }
  };
  const int lanes = D == 0 ? ch.count : NL;
  if ((int)threadIdx.x < ch.count) {
    const long long o = line_origin(B, D, ch.first + threadIdx.x);
    s_line[threadIdx.x] = o;
    s_flag[threadIdx.x] = (B.prim[o] < 0.0 ? 1 : 0) | (B.prim[o + (long long)(L + 5) * st] < 0.0 ? 2 : 0);
  }
  __syncthreads();
  {
    const S* const prim = FluxSrc<S>::prim(B);
    const S* const met = FluxSrc<S>::metrics(B);
    const S* const vol = FluxSrc<S>::vol(B);
    const S* const mu = B.mu;
    const S* const der = B.duvwt;
    for (int it = threadIdx.x; it < lanes * ns; it += blockDim.x) {
      int lane, x;
      item(it, ns, lane, x);
      if (lane >= ch.count) continue;
      const int p = fA - 2 + x;
      const long long at = s_line[lane] + (long long)(p + NG) * st;
      // the cross derivatives exist inside only: the end values stand in beyond
      const long long ac = s_line[lane] + (long long)(min(max(p, 0), L - 1) + NG) * st;
      T* const dst = Q + q_at(lane, x);
#pragma unroll
      for (int m = 0; m < 4; ++m) cp_async_value(dst + (VU + m) * QN, prim + (m < 3 ? m + 1 : 5) * np + at);
      cp_async_value(dst + VMU * QN, mu + at);
      cp_async_value(dst + VVOL * QN, vol + at);
#pragma unroll
      for (int m = 0; m < 9; ++m) cp_async_value(dst + (VMET + m) * QN, met + m * np + at);
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        cp_async_value(dst + (VX + m) * QN, der + (m + 4 * D1) * np + ac);
        cp_async_value(dst + (VX + 4 + m) * QN, der + (m + 4 * D2) * np + ac);
      }
    }
  }
  cp_async_commit();
  // the increments this thread will change, on their way meanwhile
  const int nc = ch.c1 - ch.c0;
  constexpr int NO = (Z::CM * NL + Z::NT - 1) / Z::NT;
  S old[NO][4];
#pragma unroll
  for (int o = 0; o < NO; ++o) {
    const int it = threadIdx.x + o * Z::NT;
    int lane, x;
    item(it, nc, lane, x);
    if (it < lanes * nc && lane < ch.count) {
      const S* const dq = B.dq + s_line[lane] + (long long)(ch.c0 + x + NG) * st;
#pragma unroll
      for (int m = 0; m < 4; ++m) old[o][m] = dq[(m + 1) * np];
    }
  }
  cp_async_wait<0>();
  __syncthreads();
  for (int it = threadIdx.x; it < lanes * nf; it += blockDim.x) {
    int lane, x;
    item(it, nf, lane, x);
    if (lane >= ch.count) continue;
    const int f = fA + x;
    const T* const q = Q + q_at(lane, x + 2);  // point f
    auto half = [&](int v) -> T {
      const T* const a = q + v * QN;
      return (T(9) * (a[-QS] + a[0]) + T(-1) * (a[QS] + a[-2 * QS])) / T(16);
    };
    const bool fl = (s_flag[lane] & 1) && f <= 1, fr = (s_flag[lane] & 2) && f >= L - 1;
    T uvwt[4], d[12];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const T* const a = q + (VU + m) * QN;
      uvwt[m] = (T(9) * (a[-QS] + a[0]) + T(-1) * (a[QS] + a[-2 * QS])) / T(16);
      d[m + 4 * D] = div24(T(27) * (a[0] - a[-QS]) + T(-1) * (a[QS] - a[-2 * QS]));
    }
    if (fl || fr) {  // one-sided at a flagged end: points 0.. from the low, L-1.. from the high end
      const int in = fl ? QS : -QS;
      const bool first = fl ? f == 0 : f == L;
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const T* const a = q + (VU + m) * QN + ((fl ? 0 : L - 1) - f) * QS;
        const T q1 = a[0], q2 = a[in], q3 = a[2 * in], q4 = a[3 * in];
        T g;
        if (first) {
          uvwt[m] = (T(35) * q1 + T(-35) * q2 + T(21) * q3 + T(-5) * q4) / T(16);
          g = T(-71) * q1 + T(141) * q2 + T(-93) * q3 + T(23) * q4;
        } else {
          uvwt[m] = (T(5) * q1 + T(15) * q2 + T(-5) * q3 + T(1) * q4) / T(16);
          g = T(-22) * q1 + T(17) * q2 + T(9) * q3 + T(-5) * q4 + T(1) * a[4 * in];
        }
        d[m + 4 * D] = fl ? div24(g) : -div24(g);
      }
    }
    const T vs = half(VMU);
    const T kcp = vs * cp_prl;
    const T volh = half(VVOL);
    T kxyz[9];
#pragma unroll
    for (int m = 0; m < 9; ++m) kxyz[m] = half(VMET + m);
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      d[m + 4 * D1] = half(VX + m);
      d[m + 4 * D2] = half(VX + 4 + m);
    }
    // transform_derivs_to_phys
    const T vol_inv = over(volh).r;
    T g[12];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      const T k1 = kxyz[m], k2 = kxyz[m + 3], k3 = kxyz[m + 6];
#pragma unroll
      for (int v = 0; v < 4; ++v) g[v * 3 + m] = (k1 * d[v] + k2 * d[v + 4] + k3 * d[v + 8]) * vol_inv;
    }
    // compute_viscous_flux_1d
    const T CC = T(2.0 / 3.0);
    const T vscc = vs * CC;
    const T dudx = g[0], dudy = g[1], dudz = g[2];
    const T dvdx = g[3], dvdy = g[4], dvdz = g[5];
    const T dwdx = g[6], dwdy = g[7], dwdz = g[8];
    const T txx = vscc * (T(2) * dudx - dvdy - dwdz);
    const T tyy = vscc * (T(2) * dvdy - dwdz - dudx);
    const T tzz = vscc * (T(2) * dwdz - dudx - dvdy);
    const T txy = vs * (dudy + dvdx);
    const T txz = vs * (dudz + dwdx);
    const T tyz = vs * (dvdz + dwdy);
    const T nx = kxyz[3 * D + 0], ny = kxyz[3 * D + 1], nz = kxyz[3 * D + 2];
    T* const fv = F + f_at(lane, x);
    const T f0 = txx * nx + txy * ny + txz * nz;
    const T f1 = txy * nx + tyy * ny + tyz * nz;
    const T f2 = txz * nx + tyz * ny + tzz * nz;
    const T work = uvwt[0] * f0 + uvwt[1] * f1 + uvwt[2] * f2;
    const T heat = kcp * (g[9] * nx + g[10] * ny + g[11] * nz);
    fv[0] = f0;
    fv[FN] = f1;
    fv[2 * FN] = f2;
    fv[3 * FN] = work + heat;
  }
  __syncthreads();
#pragma unroll
  for (int o = 0; o < NO; ++o) {
    const int it = threadIdx.x + o * Z::NT;
    int lane, x;
    item(it, nc, lane, x);
    if (it >= lanes * nc || lane >= ch.count) continue;
    const int t = ch.c0 + x;
    S* const dq = B.dq + s_line[lane] + (long long)(t + NG) * st;
    const T* const s = F + f_at(lane, t - fA);  // face t
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const T* const f = s + m * FN;
      const T dfv = flux_diff_at<T>([&](int k) -> T { return f[(k - t) * QS]; }, t, L);
      dq[(m + 1) * np] = (S)((T)old[o][m] - re_inv * dfv);
    }
  }
}

}  // namespace orion
