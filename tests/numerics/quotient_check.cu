// Holds the FP64 quotients of the flux kernels and sweeps to the division, bit
// for bit (signs of zeros included), on the device and with the library's own
// compiler flags: quotient() with its denominators' reciprocals, the quotients
// by 6, 12, 24 and 1920, and the WCNS states against the reference's formulas
// with one division per quotient.
// Prints "ok" or the first disagreement.
#include <cstdio>
#include <cstring>

#include "inviscid.cuh"

using namespace orion;

struct Fault {
  int what;  // 0: none
  double in[5], got, want;
};

__device__ unsigned long long draw(unsigned long long& s) {  // splitmix64
  unsigned long long z = (s += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
// A random mantissa at a random exponent of [lo, hi]; the mantissa's low bits all set or clear now and then.
__device__ double number(unsigned long long& s, int lo, int hi) {
  unsigned long long m = draw(s) & 0xfffffffffffffull;
  const unsigned long long how = draw(s) % 8;
  if (how == 0) m = 0;
  if (how == 1) m = 0xfffffffffffffull;
  if (how == 2) m &= ~0xffffffull;
  const int e = lo + (int)(draw(s) % (unsigned)(hi - lo + 1));
  return __longlong_as_double((long long)(((unsigned long long)(e + 1023) << 52) | m));
}
__device__ bool same(double a, double b) {
  return __double_as_longlong(a) == __double_as_longlong(b) || (isnan(a) && isnan(b));
}
__device__ void hold(Fault* f, int what, double got, double want, const double in[5]) {
  if (same(got, want) || atomicCAS(&f->what, 0, what) != 0) return;
  for (int m = 0; m < 5; ++m) f->in[m] = in[m];
  f->got = got;
  f->want = want;
}

__device__ double weight(double c, double g, double s) {
  const double i = 1.0e-6 + (g * g + s * s);
  return c / (i * i);
}
// InviscidFluxComputer.cpp:259-315 around point c
__device__ void states(const double q[5], double& l, double& r) {
  const double a = q[0], b = q[1], c = q[2], d = q[3], e = q[4];
  const double s1 = a - 2.0 * b + c, s2 = b - 2.0 * c + d, s3 = c - 2.0 * d + e;
  const double g1 = 0.5 * (a - 4.0 * b + 3.0 * c), g2 = 0.5 * (d - b), g3 = 0.5 * (-3.0 * c + 4.0 * d - e);
  {
    const double w1 = weight(1.0 / 16.0, g1, s1), w2 = weight(10.0 / 16.0, g2, s2), w3 = weight(5.0 / 16.0, g3, s3);
    const double sum = w1 + w2 + w3;
    l = c + 0.125 * ((w1 / sum) * (s1 + 4.0 * g1) + (w2 / sum) * (s2 + 4.0 * g2) + (w3 / sum) * (s3 + 4.0 * g3));
  }
  {
    const double w1 = weight(5.0 / 16.0, g1, s1), w2 = weight(10.0 / 16.0, g2, s2), w3 = weight(1.0 / 16.0, g3, s3);
    const double sum = w1 + w2 + w3;
    r = c + 0.125 * ((w1 / sum) * (s1 - 4.0 * g1) + (w2 / sum) * (s2 - 4.0 * g2) + (w3 / sum) * (s3 - 4.0 * g3));
  }
}

__global__ void k_check(Fault* f, int rounds) {
  unsigned long long s = 0x5851F42D4C957F2Dull * (blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x + 1);
  const double inf = __longlong_as_double(0x7ff0000000000000ll);
  for (int it = 0; it < rounds; ++it) {
    // exponents wide and near one; now and then a zero, an infinity or a NaN
    const bool near = draw(s) & 1;
    double a = near ? number(s, -30, 30) : number(s, -959, 1022);
    const double b = near ? number(s, -30, 30) : number(s, -959, 959);
    const unsigned long long how = draw(s) % 32;
    if (how == 0) a = 0.0;
    if (how == 1) a = inf;
    if (how == 2) a = inf - inf;
    if (how == 3) a = b;
    if (how == 4) a = number(s, -2, 2) * b;
    if (draw(s) & 1) a = -a;
    const double in[5] = {a, b, 0, 0, 0};
    const double q = a / b;
    // a quotient below the normal range may differ in its last bit
    if (!(q != 0.0 && fabs(q) < 2.2250738585072014e-308) && !(a != 0.0 && q == 0.0)) {
      hold(f, 1, div(a, over(b)), q, in);
      hold(f, 2, quotient(a, b, quotient_rcp(b)), q, in);
    }
    hold(f, 3, div6(a), a / 6.0, in);
    hold(f, 4, div12(a), a / 12.0, in);
    hold(f, 5, div24(a), a / 24.0, in);
    hold(f, 6, div1920(a), a / 1920.0, in);
    // a denominator or numerator of infinity, a zero denominator
    const double edge[5] = {a, how & 1 ? inf : 0.0, 0, 0, 0};
    if (how < 8) hold(f, 7, div(a, over(edge[1])), a / edge[1], edge);
    // line values: alike, smooth, jumping, of any size up to 1e60
    double p[5];
    const double base = number(s, draw(s) & 1 ? -3 : -190, draw(s) & 1 ? 3 : 190);
    for (int m = 0; m < 5; ++m) {
      const unsigned long long k = draw(s) % 4;
      p[m] = k == 0 ? base : (k == 1 ? base * (1.0 + number(s, -30, -1)) : (k == 2 ? number(s, -3, 3) : -base));
      if (how < 4) p[m] = base;
    }
    double l, r, wl, wr;
    wcns_states(p[0], p[1], p[2], p[3], p[4], l, r);
    states(p, wl, wr);
    hold(f, 8, l, wl, p);
    hold(f, 9, r, wr, p);
  }
}

int main() {
  Fault* d = nullptr;
  Fault f;
  std::memset(&f, 0, sizeof(f));
  if (cudaMalloc(&d, sizeof(f)) != cudaSuccess || cudaMemcpy(d, &f, sizeof(f), cudaMemcpyHostToDevice) != cudaSuccess) return 2;
  k_check<<<148, 256>>>(d, 2000);
  if (cudaMemcpy(&f, d, sizeof(f), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  if (f.what == 0) {
    std::printf("ok\n");
    return 0;
  }
  static const char* const names[] = {"", "div", "quotient, quotient_rcp", "div6", "div12", "div24", "div1920",
                                      "div by an infinity or zero", "left state", "right state"};
  std::printf("%s: %a %a %a %a %a gives %a, not %a\n", names[f.what], f.in[0], f.in[1], f.in[2], f.in[3], f.in[4], f.got, f.want);
  return 1;
}
