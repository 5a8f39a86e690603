// Inviscid RHS along one direction (compute_block_inviscid + compute_flux_line,
// src/solver/InviscidFluxComputer.cpp:136-192, 238-522, 543-647).
//
// A CTA takes NL neighbouring grid lines of one block and a chunk of points
// along them, in three phases through shared memory:
//   points  the WCNS-E-5 left and right states of every point of the chunk.
//           The smoothness measures of a point are the same for the state on
//           either side of it, so forming both at once halves them, and the
//           weights share reciprocals;
//   faces   boundary stencils, positivity fallback and the Roe flux, and at a
//           flagged line end the 13 fluxes of the boundary re-calculation
//           rounds (:377-521), one thread each;
//   output  the flux difference, or at the three points of a flagged end the
//           rounds' sums, added to dq.
// What bounds it: the phases' latency.  Neither pipe is full (193x97x65: an
// instruction issues in 57-62% of the cycles in FP32 and 42-46% in FP64, the
// FP64 pipe works in 40-44%), and the first stall is the barrier between the
// phases, with four (FP32) or three CTAs an SM to fill in for one another.
// Each prim and metric value is read from global memory once per chunk into
// shared memory (a face used to read 30 and 12, with their addresses).  A
// chunk needs two or three faces more than points on each inner side, so lines
// are cut into as few, even chunks as the buffers hold; chunks of 32 (64 along
// i) leave room for four CTAs an SM in FP32, and that is worth more than the
// repeated faces: 385x257x129 in 64 blocks, the three directions, mixed 2.19 ms
// (48 points and three CTAs 2.35), plain 6.61 (7.07); half the lines and
// threads 2.61 and 7.80.  One thread a face over whole lines, with the rounds
// in kernels of their own, took 3.23 and 12.0.
#pragma once

#include "device_types.cuh"
#include "numerics.cuh"
#include "kernels.cuh"

namespace orion {

// Lines per CTA (64-byte rows across the lines; along i the points are the
// contiguous direction) and points per chunk.
template <int D, typename T> struct InvShape {
  static constexpr int NL = (D == 0 ? 4 : 8) * 8 / (int)sizeof(T);
  static constexpr int CM = D == 0 ? 64 : 32;
  static constexpr int NT = 256;
  static constexpr int NS = CM + 10;  // staged points: stencils of the chunk's states
  static constexpr int NP = CM + 6;   // points with states
  static constexpr size_t smem = sizeof(T) * NL * ((size_t)8 * NS + 10 * NP + 2 * 13 * 5);
};

// One state on either side of point c from the five points around it: l
// towards d, r towards b (:259-315).  FP64 reproduces the reference's operations:
// C / D with C = 1/16 is the reciprocal scaled exactly, the other quotients go
// through quotient() from the shared reciprocal.
__device__ __forceinline__ void wcns_states(double a, double b, double c, double d, double e, double& l, double& r) {
  const double CL1 = 1.0 / 16.0, CL2 = 10.0 / 16.0, CL3 = 5.0 / 16.0, EPS = 1.0e-6;
  const double s1 = a - 2.0 * b + c, s2 = b - 2.0 * c + d, s3 = c - 2.0 * d + e;
  const double g1 = 0.5 * (a - 4.0 * b + 3.0 * c), g2 = 0.5 * (d - b), g3 = 0.5 * (-3.0 * c + 4.0 * d - e);
  const double i1 = EPS + (g1 * g1 + s1 * s1), i2 = EPS + (g2 * g2 + s2 * s2), i3 = EPS + (g3 * g3 + s3 * s3);
  const double d1 = i1 * i1, d2 = i2 * i2, d3 = i3 * i3;
  const double r1 = __drcp_rn(d1), r3 = __drcp_rn(d3);
  const double w2 = CL2 / d2;
  const double x1 = s1 + 4.0 * g1, x2 = s2 + 4.0 * g2, x3 = s3 + 4.0 * g3;
  {
    const double w1 = CL1 * r1, w3 = quotient(CL3, d3, r3);
    const double sum = w1 + w2 + w3, rs = __drcp_rn(sum);
    l = c + 0.125 * (quotient(w1, sum, rs) * x1 + quotient(w2, sum, rs) * x2 + quotient(w3, sum, rs) * x3);
  }
  const double y1 = s1 - 4.0 * g1, y2 = s2 - 4.0 * g2, y3 = s3 - 4.0 * g3;
  {
    const double w1 = quotient(CL3, d1, r1), w3 = CL1 * r3;
    const double sum = w1 + w2 + w3, rs = __drcp_rn(sum);
    r = c + 0.125 * (quotient(w1, sum, rs) * y1 + quotient(w2, sum, rs) * y2 + quotient(w3, sum, rs) * y3);
  }
}
__device__ __forceinline__ void wcns_states(float a, float b, float c, float d, float e, float& l, float& r) {
  const float s1 = a - 2.f * b + c, s2 = b - 2.f * c + d, s3 = c - 2.f * d + e;
  const float g1 = 0.5f * (a - 4.f * b + 3.f * c), g2 = 0.5f * (d - b), g3 = 0.5f * (-3.f * c + 4.f * d - e);
  const float i1 = 1.0e-6f + (g1 * g1 + s1 * s1), i2 = 1.0e-6f + (g2 * g2 + s2 * s2), i3 = 1.0e-6f + (g3 * g3 + s3 * s3);
  const float r1 = __fdividef(1.f, i1 * i1), r2 = __fdividef(10.f, i2 * i2), r3 = __fdividef(1.f, i3 * i3);
  const float l3 = 5.f * r3, q1 = 5.f * r1;
  l = c + __fdividef(0.125f, r1 + r2 + l3) * (r1 * (s1 + 4.f * g1) + r2 * (s2 + 4.f * g2) + l3 * (s3 + 4.f * g3));
  r = c + __fdividef(0.125f, q1 + r2 + r3) * (q1 * (s1 - 4.f * g1) + r2 * (s2 - 4.f * g2) + r3 * (s3 - 4.f * g3));
}

// The fluxes of the boundary re-calculation rounds of one flagged line end
// (:377-521): face (counted from the end), the near and the far state as
// combinations of the four points nearest the end, the coefficient in the
// output's sum, and the output (0, 1, 2 from the end).  near_ is the left state
// at the low end of a line and the right state at the high end.  far den 0:
// the far state is the face's own WCNS state.
struct RoundFlux {
  signed char face, out;
  short coef;
  short near_[4], near_den;
  short far_[4], far_den;
};
static __device__ __constant__ RoundFlux kRounds[13] = {
    {0, 0, -23, {3, -1, 0, 0}, 2, {3, -1, 0, 0}, 2},
    {1, 0, 21, {19, 25, -2, 0}, 42, {19, 25, -2, 0}, 42},
    {2, 0, 3, {4, 3, 9, 2}, 18, {4, 3, 9, 2}, 18},
    {3, 0, -1, {-2, 3, 3, 2}, 6, {-2, 3, 3, 2}, 6},
    {1, 1, -22, {3, 6, -1, 0}, 8, {3, 6, -1, 0}, 8},
    {2, 1, 17, {-30, 145, 29, -8}, 136, {2, 49, 125, -40}, 136},
    {3, 1, 9, {0, -1, 6, 3}, 8, {0, -1, 6, 3}, 8},
    {4, 1, -5, {0, 1, 2, 5}, 8, {0, 1, 2, 5}, 8},
    {5, 1, 1, {0, 1, 1, 6}, 8, {0, 1, 1, 6}, 8},
    {1, 2, 1, {3, 6, -1, 0}, 8, {5, 15, -5, 1}, 16},
    {2, 2, -27, {-29, 170, 63, 12}, 216, {0, 0, 0, 0}, 0},
    {3, 2, 27, {0, -1, 6, 3}, 8, {0, 0, 0, 0}, 0},
    {4, 2, -1, {0, 1, 2, 5}, 8, {0, 0, 0, 0}, 0},
};

// (c0 q0 + c1 q1 + c2 q2 + c3 q3) / den, terms with a zero coefficient left out.
template <typename T>
__device__ __forceinline__ T round_state(const short c[4], short den, const T q[4]) {
  T s = T(0);
#pragma unroll
  for (int x = 0; x < 4; ++x) {
    const T t = T(c[x]) * q[x];
    if (c[x] != 0) s = s + t;
  }
  return s / T(den);
}

template <int D, typename S, typename T>
__global__ void __launch_bounds__(256, LineMinBlocks<T>::inv) k_inviscid(const BlockDev<S>* __restrict__ blocks,
                                                                         const LineChunk* __restrict__ chunks) {
  using Z = InvShape<D, T>;
  constexpr int NL = Z::NL, NS = Z::NS, NP = Z::NP;
  constexpr int QS = D == 0 ? 1 : NL;                     // step along the line in shared memory
  constexpr int QN = NS * NL, PN = NP * NL;               // one staged variable, one state variable
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* const Q = reinterpret_cast<T*>(smem_raw);            // prim 5, metrics 3
  T* const ST = Q + 8 * QN;                               // left states 5 (then fluxes of the face above), right states 5
  T* const BF = ST + 10 * PN;                             // rounds: [end][flux][component][line]
  __shared__ unsigned char s_flag[NL];
  __shared__ long long s_line[NL];  // line origins
  const LineChunk ch = chunks[blockIdx.x];
  const BlockDev<S>& B = blocks[ch.block];
  const long long np = B.npad;
  const int L = dim_along(B, D);
  const long long st = stride_along(B, D);
  const T gamma = T(B.prm.gamma);
  const int fA = max(0, ch.c0 - 2), fB = min(L, ch.c1 + 2);  // faces
  const int nf = fB - fA + 1, ns = nf + 5, npt = nf + 1;     // staged points from fA - 3, states from fA - 1
  auto q_at = [&](int lane, int x) { return D == 0 ? lane * NS + x : x * NL + lane; };
  auto p_at = [&](int lane, int x) { return D == 0 ? lane * NP + x : x * NL + lane; };
  auto item = [&](int it, int n, int& lane, int& x) {
    if (D == 0) {
      lane = it / n;
      x = it - lane * n;
    } else {
      x = it / NL;
      lane = it - x * NL;
    }
  };
  const int lanes = D == 0 ? ch.count : NL;  // lines the loops run over (along j and k idle ones too)
  if ((int)threadIdx.x < ch.count) {
    const long long o = line_origin(B, D, ch.first + threadIdx.x);
    s_line[threadIdx.x] = o;
    s_flag[threadIdx.x] = (B.prim[o] < 1.0e-20 ? 1 : 0) | (B.prim[o + (long long)(L + 5) * st] < 1.0e-20 ? 2 : 0);
  }
  __syncthreads();
  {
    const S* const prim = FluxSrc<S>::prim(B);
    const S* const met = FluxSrc<S>::metrics(B) + (long long)(3 * D) * np;
    for (int it = threadIdx.x; it < lanes * ns; it += blockDim.x) {
      int lane, x;
      item(it, ns, lane, x);
      if (lane >= ch.count) continue;
      const long long at = s_line[lane] + (long long)(fA - 3 + NG + x) * st;
      T* const dst = Q + q_at(lane, x);
#pragma unroll
      for (int m = 0; m < 5; ++m) cp_async_value(dst + m * QN, prim + m * np + at);
#pragma unroll
      for (int m = 0; m < 3; ++m) cp_async_value(dst + (5 + m) * QN, met + m * np + at);
    }
  }
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  // states: point fA - 1 + x is staged at x + 2
  for (int it = threadIdx.x; it < lanes * npt; it += blockDim.x) {
    int lane, x;
    item(it, npt, lane, x);
    if (lane >= ch.count) continue;
    const T* const q = Q + q_at(lane, x + 2);
    T* const s = ST + p_at(lane, x);
    // FP64: one variable's code, or the instruction cache does not hold the loop
#pragma unroll(sizeof(T) == 8 ? 1 : 5)
    for (int m = 0; m < 5; ++m) {
      T l, r;
      wcns_states(q[m * QN - 2 * QS], q[m * QN - QS], q[m * QN], q[m * QN + QS], q[m * QN + 2 * QS], l, r);
      s[m * PN] = l;
      s[(5 + m) * PN] = r;
    }
  }
  __syncthreads();
  // metric component of face f (interp_metrics_half, :136-192, ni > 2); interior
  // point p is staged at p - fA + 3
  auto face_metric = [&](const T* q, int f) -> T {  // q: the component at point f of this line
    auto P = [&](int p) -> T { return q[(p - f) * QS]; };
    if (f == 0) return (T(35) * P(0) + T(-35) * P(1) + T(21) * P(2) + T(-5) * P(3)) / T(16);
    if (f == 1) return (T(5) * P(0) + T(15) * P(1) + T(-5) * P(2) + T(1) * P(3)) / T(16);
    if (f == L) return (T(35) * P(L - 1) + T(-35) * P(L - 2) + T(21) * P(L - 3) + T(-5) * P(L - 4)) / T(16);
    if (f == L - 1) return (T(5) * P(L - 1) + T(15) * P(L - 2) + T(-5) * P(L - 3) + T(1) * P(L - 4)) / T(16);
    return (T(9) * (P(f - 1) + P(f)) + T(-1) * (P(f + 1) + P(f - 2))) / T(16);
  };
  // The increments this thread will add to, asked for before the fluxes: the
  // loads are back by the output phase.
  const int nc = ch.c1 - ch.c0;
  constexpr int NO = (Z::CM * NL + Z::NT - 1) / Z::NT;
  S old[NO][5];
#pragma unroll
  for (int o = 0; o < NO; ++o) {
    const int it = threadIdx.x + o * Z::NT;
    int lane, x;
    item(it, nc, lane, x);
    if (it < lanes * nc && lane < ch.count) {
      const S* const dq = B.dq + s_line[lane] + (long long)(ch.c0 + x + NG) * st;
#pragma unroll
      for (int m = 0; m < 5; ++m) old[o][m] = dq[m * np];
    }
  }
  // Fluxes: first the rounds' at flagged ends inside this chunk (they read left
  // states that the faces overwrite), then the faces'; one code for both.
  const bool lo = ch.c0 == 0, hi = ch.c1 == L;
#pragma unroll 1
  for (int faces = 0; faces < 2; ++faces) {
    const int items = faces ? lanes * nf : (lo || hi ? 2 * 13 * NL : 0);
#pragma unroll 1
    for (int it = threadIdx.x; it < items; it += blockDim.x) {
      int lane, f;
      T ql[5], qr[5], out[5];
      T* dst;
      int ds;
      if (faces) {
        int x;
        item(it, nf, lane, x);
        if (lane >= ch.count) continue;
        // face fA + x has the left state of state point x and the right one of x + 1
        f = fA + x;
        T* const s = ST + p_at(lane, x);
        dst = s;
        ds = PN;
#pragma unroll
        for (int m = 0; m < 5; ++m) {
          ql[m] = s[m * PN];
          qr[m] = s[(5 + m) * PN + QS];
        }
        const int flag = s_flag[lane];
        if ((flag & 1) && f <= 2) {  // fixed stencils of a flagged low end
          const T* const q = Q + q_at(lane, 3 - fA);
#pragma unroll
          for (int m = 0; m < 5; ++m) {
            const T q1 = q[m * QN], q2 = q[m * QN + QS], q3 = q[m * QN + 2 * QS], q4 = q[m * QN + 3 * QS];
            if (f == 0) ql[m] = qr[m] = (T(35.) * q1 - T(35.) * q2 + T(21.) * q3 - T(5.) * q4) / T(16.);
            else if (f == 1) ql[m] = qr[m] = (T(5.) * q1 + T(15.) * q2 - T(5.) * q3 + q4) / T(16.);
            else ql[m] = (-q1 + T(9.) * q2 + T(9.) * q3 - q4) / T(16.);
          }
        }
        if ((flag & 2) && f >= L - 2) {
          const T* const q = Q + q_at(lane, L - 1 - fA + 3);
#pragma unroll
          for (int m = 0; m < 5; ++m) {
            const T qn = q[m * QN], qn1 = q[m * QN - QS], qn2 = q[m * QN - 2 * QS], qn3 = q[m * QN - 3 * QS];
            if (f == L) ql[m] = qr[m] = (T(35.) * qn - T(35.) * qn1 + T(21.) * qn2 - T(5.) * qn3) / T(16.);
            else if (f == L - 1) ql[m] = qr[m] = (T(5.) * qn + T(15.) * qn1 - T(5.) * qn2 + qn3) / T(16.);
            else qr[m] = (-qn + T(9.) * qn1 + T(9.) * qn2 - qn3) / T(16.);
          }
        }
      } else {
        const int end = it / (13 * NL), r = it - end * (13 * NL), e = r / NL;
        lane = r - e * NL;
        if (lane >= ch.count || !(end ? hi : lo) || !(s_flag[lane] & (1 << end))) continue;
        const RoundFlux& R = kRounds[e];
        f = end ? L - R.face : R.face;
        dst = BF + (end * 13 + e) * 5 * NL + lane;
        ds = NL;
        const T* const q = Q + q_at(lane, (end ? L - 1 : 0) - fA + 3);  // the end's point
        const int in = end ? -QS : QS;
#pragma unroll
        for (int m = 0; m < 5; ++m) {
          const T p[4] = {q[m * QN], q[m * QN + in], q[m * QN + 2 * in], q[m * QN + 3 * in]};
          const T n = round_state<T>(R.near_, R.near_den, p);
          T o;
          if (R.far_den) o = round_state<T>(R.far_, R.far_den, p);
          else o = end ? ST[m * PN + p_at(lane, f - fA)] : ST[(5 + m) * PN + p_at(lane, f - fA + 1)];
          ql[m] = end ? o : n;
          qr[m] = end ? n : o;
        }
      }
      // positivity fallback + Roe flux at face f (calc_flux_loop, :342-364)
      const T* const q = Q + q_at(lane, f - fA + 3);  // point f
      if (ql[0] <= T(1e-6) || ql[4] <= T(1e-6)) {
        const int p = max(f - 1, 0) - 1;
#pragma unroll
        for (int m = 0; m < 5; ++m) ql[m] = q[m * QN + (p - f) * QS];
      }
      if (qr[0] <= T(1e-6) || qr[4] <= T(1e-6)) {
        const int p = min(L - 1, f);
#pragma unroll
        for (int m = 0; m < 5; ++m) qr[m] = q[m * QN + (p - f) * QS];
      }
      T k[3];
#pragma unroll
      for (int m = 0; m < 3; ++m) k[m] = face_metric(q + (5 + m) * QN, f);
      roe_flux<T>(ql, qr, k[0], k[1], k[2], T(0), T(0.1), gamma, out);
#pragma unroll
      for (int m = 0; m < 5; ++m) dst[m * ds] = out[m];
    }
    __syncthreads();
  }
  // dq += flux difference; at a flagged end's three points the rounds' sums
#pragma unroll
  for (int o = 0; o < NO; ++o) {
    const int it = threadIdx.x + o * Z::NT;
    int lane, x;
    item(it, nc, lane, x);
    if (it >= lanes * nc || lane >= ch.count) continue;
    const int t = ch.c0 + x, flag = s_flag[lane];
    S* const dq = B.dq + s_line[lane] + (long long)(t + NG) * st;
    const bool rl = (flag & 1) && t <= 2, rh = (flag & 2) && t >= L - 3;
    if (rl || rh) {
      const int out = rl ? t : L - 1 - t;
      const int e0 = out == 0 ? 0 : (out == 1 ? 4 : 9), n = out == 1 ? 5 : 4;
#pragma unroll
      for (int m = 0; m < 5; ++m) {
        const T* const b = BF + (((rl ? 0 : 13) + e0) * 5 + m) * NL + lane;
        T acc = T(kRounds[e0].coef) * b[0];
        for (int e = 1; e < n; ++e) acc = acc + T(kRounds[e0 + e].coef) * b[e * 5 * NL];
        if (rh && !rl) acc = -acc;
        dq[m * np] = (S)((T)old[o][m] + div24(acc));
      }
      continue;
    }
    const T* const s = ST + p_at(lane, t - fA);  // face t
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      const T* const f = s + m * PN;
      dq[m * np] = (S)((T)old[o][m] + flux_diff_at<T>([&](int k) -> T { return f[(k - t) * QS]; }, t, L));
    }
  }
}

}  // namespace orion
