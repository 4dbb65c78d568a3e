// The pieces of the on-the-fly coefficients (qg_coef.cuh) compiled for the host
// and compared with binary128: the reciprocal, the phase, and the Lagrange
// weights of both precisions.  u = 2^-53 (FP32: 2^-24).  Exit status 1 on any
// value past its bound.
#include <quadmath.h>

#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>

#include <vector_functions.h>
#undef __device__
#define __device__
#undef __forceinline__
#define __forceinline__ inline
static float __int_as_float(int i)
{
  float f;
  std::memcpy(&f, &i, 4);
  return f;
}
static void sincospi(double x, double *s, double *c) { *s = (double)sinq(M_PIq * x), *c = (double)cosq(M_PIq * x); }
static void sincospif(float x, float *s, float *c) { *s = (float)sinq(M_PIq * x), *c = (float)cosq(M_PIq * x); }

#include "../../quest_b200/csrc/qg_coef.cuh"

typedef __float128 qf;
static int bad = 0;
static double worst[6];  // largest error over its bound, by check

static void expect(int check, const char *what, qf error, qf bound, double at)
{
  const double r = (double)(fabsq(error) / bound);
  if(r > worst[check]) worst[check] = r;
  if(!(r <= 1.0) && ++bad < 10) std::printf("%s at %.17g: %.3f of its bound\n", what, at, r);
}

// Weights at the fraction x.  The rounded pieces are f_m = x - m (u each) and
// their reciprocals (2 u more), so with n = q + 4 roundings on any path:
//   w0          2 (q + 2) u relative (q factors, their products, 1/den);
//   d1          n u S1, S1 = sum 1/|f_m|;
//   d2 + d1^2   4 n u S1^2 (d1^2 twice its error, sum of squares S2 <= S1^2);
//   jets        (3 q + 4) u times the polynomial of the factors' sizes.
template <int Q>
static void weights(double x)
{
  const double u = 0x1p-53, uf = 0x1p-24;
  const float xf = (float)x;
  qg::lagrange_taps<Q>(x, [&](int b, double w0, double d1, double s2) {
    qf w = 1, d = 0, e = 0, S1 = 0;
    for(int m = 0; m <= Q; ++m)
      if(m != b) {
        const qf f = (qf)x - m;
        w *= f / (b - m), d -= 1 / f, e -= 1 / (f * f), S1 += fabsq(1 / f);
      }
    expect(1, "w0", w0 - w, 2 * (Q + 2) * u * fabsq(w), x);
    expect(2, "d1", d1 - d, (Q + 4) * u * S1, x);
    expect(3, "d2 + d1^2", s2 - (e + d * d), 4 * (Q + 4) * u * S1 * S1, x);
  });
  qg::lagrange_jets<Q>(xf, [&](int b, const qg::Jet<float> &j) {
    qf v = 1, d = 0, h = 0, V = 1, D = 0, H = 0;
    for(int m = 0; m <= Q; ++m)
      if(m != b) {
        const qf f = (qf)xf - m, F = fabsq(f);
        h = h * f + d, d = d * f + v, v = v * f;
        H = H * F + D, D = D * F + V, V = V * F;
      }
    const qf k = (3 * Q + 4) * uf;
    expect(4, "jet value", j.v - v, k * V + FLT128_MIN, x);
    expect(4, "jet derivative", j.d - d, k * D + FLT128_MIN, x);
    expect(4, "jet second derivative", j.h - h, k * H + FLT128_MIN, x);
  });
}

int main()
{
  std::mt19937_64 gen(7);
  std::uniform_real_distribution<double> unit(0.0, 1.0);
  for(int i = 0; i < 400000; ++i) {
    // any approximation within 2^-20, at its ends too
    const double x = std::ldexp(1.0 + unit(gen), (int)(gen() % 120) - 60) * (gen() & 1 ? 1 : -1);
    const double off = i % 3 == 0 ? 1.0 : i % 3 == 1 ? -1.0 : 2 * unit(gen) - 1;
    const double y = (double)((1 + (qf)off * 0x1.fp-21) / x);
    expect(0, "reciprocal", qg::rcp_refine(x, y) * (qf)x - 1, 0x1p-53 * (1 + 0x1p-6), x);
  }
  for(int i = 0; i < 400000; ++i) {
    qg_params p{};
    p.hbar = p.mu0 = 1, p.dt = 1e-3;
    p.c0 = i & 1 ? 1.0 : 100 * (1 + unit(gen));
    p.laser_frequency = 2000 * unit(gen) + 1;
    const qg::OtfConst o = qg::otf_const(p);
    const double r = unit(gen);
    const qf exact = (qf)p.laser_frequency * r / (M_PIq * (qf)p.c0);
    expect(5, "phase", qg::half_turns(r, o) - exact, 0x1p-53 * (1 + 0x1p-9) * exact, r);
  }
  for(int i = 0; i < 30000; ++i) {
    const double t = unit(gen), x = i % 4 == 0 ? t * 1e-4 + 1e-12 : i % 4 == 1 ? 1 - t * 1e-4 - 1e-12 : t;
    weights<1>(x), weights<2>(x), weights<3>(x), weights<4>(x), weights<5>(x), weights<6>(x), weights<7>(x);
  }
  std::printf("largest errors over their bounds: 1/x %.3f, w0 %.3f, d1 %.3f, d2 + d1^2 %.3f, jets %.3f, phase %.3f\n",
              worst[0], worst[1], worst[2], worst[3], worst[4], worst[5]);
  std::printf("mismatches %d\n", bad);
  return bad != 0;
}
