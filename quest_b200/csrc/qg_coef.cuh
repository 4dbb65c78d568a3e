// Per-pair retarded-interaction coefficients on the device, following the
// reference's table build operation by operation:
//   separation / norm / split_double   history_interaction.cpp:29-35, 88-97
//   UniformLagrangeSet::calculate_weights   lagrange_set.cpp:17-41
//   spatial dyads                      green_function.h:32-55
//   RotatingDyadic::coefficients       rotating_green_function.cpp:3-24
//   Dyadic::coefficients (lab frame)   green_function.cpp:3-20
//   d_obs . (M d_src)                  history_interaction.cpp:40-43
// Included by translation units compiled with -fmad=false, so each multiply
// and add rounds separately as in the reference's x86-64 build.
#pragma once

#include "qg_internal.h"

namespace qg {

// lagrange_set.cpp:17-41; w[k][i] for derivative k = 0..2, node i = 0..q.
template <int Q>
__device__ __forceinline__ void lagrange_weights_ref(double x, double dt, double (&w)[3][Q + 1])
{
#pragma unroll
  for(int b = 0; b <= Q; ++b) {
    double d0 = 1, d1 = 0, d2 = 0;
#pragma unroll
    for(int m = 0; m <= Q; ++m) {
      if(m == b) continue;
      d0 *= (x - m) / (double)(b - m);
      d1 -= 1 / (x - m);
      d2 -= pow(x - m, -2.0);
    }
    w[0][b] = d0;
    w[1][b] = w[0][b] * d1;
    w[2][b] = w[0][b] * d2 + (w[1][b] * w[1][b]) / w[0][b];
  }
  const double inv_dt = 1.0 / dt;  // gcc folds pow(dt, -1) to 1/dt
  const double inv_dt2 = pow(dt, -2.0);
#pragma unroll
  for(int i = 0; i <= Q; ++i) {
    w[1][i] *= inv_dt;
    w[2][i] *= inv_dt2;
  }
}

__device__ __forceinline__ double2 cmul(double2 a, double2 b)
{
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b)
{
  return make_double2(a.x + b.x, a.y + b.y);
}
__device__ __forceinline__ double2 cscale(double2 a, double s)
{
  return make_double2(a.x * s, a.y * s);
}

// d_obs . (M d_src) with Eigen's left-to-right sums over 3-vectors.
__device__ __forceinline__ double2 contract3(const double (&dobs)[3], const double2 (&M)[9],
                                             const double (&dsrc)[3])
{
  double2 v[3];
#pragma unroll
  for(int r = 0; r < 3; ++r) {
    double2 acc = cscale(M[3 * r + 0], dsrc[0]);
    acc = cadd(acc, cscale(M[3 * r + 1], dsrc[1]));
    acc = cadd(acc, cscale(M[3 * r + 2], dsrc[2]));
    v[r] = acc;
  }
  double2 out = cscale(v[0], dobs[0]);
  out = cadd(out, cscale(v[1], dobs[1]));
  out = cadd(out, cscale(v[2], dobs[2]));
  return out;
}

// Floor delay and q+1 coefficients of the pair (src = larger user index,
// obs = smaller), exactly the quantities build_coefficient_table stores.
template <int Q>
__device__ __forceinline__ int pair_coef_ref(const double (&psrc)[3], const double (&pobs)[3],
                                             const double (&dsrc)[3], const double (&dobs)[3],
                                             const CoefParams &p, double2 (&coef)[Q + 1])
{
  double dr[3];
#pragma unroll
  for(int k = 0; k < 3; ++k) dr[k] = pobs[k] - psrc[k];
  const double sq = (dr[0] * dr[0] + dr[1] * dr[1]) + dr[2] * dr[2];
  const double nrm = sqrt(sq);
  double idelay;
  const double frac = modf(nrm / (p.c0 * p.dt), &idelay);
  const int fd = (int)idelay;

  double w[3][Q + 1];
  lagrange_weights_ref<Q>(frac, p.dt, w);

  // spatial dyads (green_function.h:32-40)
  double dy[3][9];
  const double c2 = p.c0 * p.c0;       // pow(c, 2)
  const double n3 = pow(nrm, 3.0);     // pow(|r|, 3)
#pragma unroll
  for(int r = 0; r < 3; ++r) {
#pragma unroll
    for(int k = 0; k < 3; ++k) {
      const double rhat = (dr[r] * dr[k]) / sq;
      const double id = (r == k) ? 1.0 : 0.0;
      const double i3 = id - 3 * rhat;
      const double i1 = id - rhat;
      dy[0][3 * r + k] = (i3 * c2) / n3;
      dy[1][3 * r + k] = (i3 * p.c0) / sq;
      dy[2][3 * r + k] = i1 / nrm;
    }
  }
  const double A = p.mu0 / (4 * M_PI * p.hbar);

  if(p.frame == 0) {
    const double om = p.omega;
    const double y = (-om * nrm) / p.c0;
    double sn, cs;
    sincos(y, &sn, &cs);
    const double2 s = make_double2(-A * cs, -A * sn);
    const double om2 = om * om;
#pragma unroll
    for(int i = 0; i <= Q; ++i) {
      const double w0 = w[0][i], w1 = w[1][i], w2 = w[2][i];
      const double2 t1 = make_double2(w1, om * w0);
      const double2 t2 = make_double2(w2 - om2 * w0, (2.0 * om) * w1);
      double2 M[9];
#pragma unroll
      for(int e = 0; e < 9; ++e) {
        const double2 a = make_double2(dy[0][e] * w0, 0.0);
        const double2 b = cmul(make_double2(dy[1][e], 0.0), t1);
        const double2 c = cmul(make_double2(dy[2][e], 0.0), t2);
        M[e] = cmul(s, cadd(cadd(a, b), c));
      }
      coef[i] = contract3(dobs, M, dsrc);
    }
  } else {
#pragma unroll
    for(int i = 0; i <= Q; ++i) {
      double2 M[9];
#pragma unroll
      for(int e = 0; e < 9; ++e) {
        double2 acc = make_double2(0.0, 0.0);
#pragma unroll
        for(int term = 0; term < 3; ++term) {
          const double2 t = make_double2((A * dy[term][e]) * w[term][i], (A * 0.0) * w[term][i]);
          acc = cadd(acc, t);
        }
        M[e] = acc;
      }
      coef[i] = contract3(dobs, M, dsrc);
    }
  }
  return fd;
}

// ---- coefficients computed in the far kernel -----------------------------------
// x / t given y = 1/t correctly rounded: q0 = x*y, the remainder x - q0*t
// exact in one fused multiply-add, then q0 + r*y rounded once.  This is
// Markstein's correction step (P. W. Markstein, IBM J. Res. Develop. 34(1),
// 1990): with y within half an ulp of 1/t and q0 within one ulp of x/t it
// returns the correctly rounded quotient, i.e. exactly x / t, barring
// underflow and overflow.  r == 0 means q0 is exact (and keeps the sign of a
// zero quotient).  Four independent divisions per evaluation become twelve
// independent flops instead of four serial division sequences.
__device__ __forceinline__ double div_by(double x, double t, double y)
{
  const double q0 = x * y;
  const double r = fma(-q0, t, x);
  return r == 0.0 ? q0 : fma(r, y, q0);
}

// 1 / x: the hardware's approximation y, whose error is 2^-20 or less, and one
// step of the third-order hyperpower iteration (M. Altman, Pacific J. Math. 10,
// 1960), y (1 + e + e^2) with e = 1 - x y, which leaves e^3.  With the last
// multiply-add's rounding the error is 2^-53 (1 + 2^-6) at most.
__device__ __forceinline__ double rcp_refine(double x, double y)
{
  const double e = fma(-x, y, 1.0);
  return fma(fma(e, e, e), y, y);
}
__device__ __forceinline__ double rcp_newton(double x)
{
  double y;
#ifdef __CUDA_ARCH__
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
#else
  y = (double)(float)(1.0 / x);  // host tests
#endif
  return rcp_refine(x, y);
}

// omega r / (pi c0), the phase in half turns, to half an ulp: the constant's
// low part takes its rounding out.
__device__ __forceinline__ double half_turns(double r, const OtfConst &o)
{
  return fma(r, o.half_turns, r * o.half_turns_low);
}

// Separation, floor delay and fraction of a pair, with the operations of
// pair_coef_ref (and of the near-pair search), so the far / mid split is the
// table's; the division by c0 dt is div_by's, the same quotient.
struct PairGeom {
  double dr[3], sq, nrm, x;
  int fd;
};
__device__ __forceinline__ PairGeom pair_geom(const double (&pa)[3], const double (&pb)[3], const OtfConst &o)
{
  PairGeom g;
#pragma unroll
  for(int k = 0; k < 3; ++k) g.dr[k] = pa[k] - pb[k];
  g.sq = (g.dr[0] * g.dr[0] + g.dr[1] * g.dr[1]) + g.dr[2] * g.dr[2];
  g.nrm = sqrt(g.sq);
  const double late = div_by(g.nrm, o.c0dt, o.inv_c0dt);
  const double idelay = trunc(late);
  g.x = late - idelay;
  g.fd = (int)idelay;
  return g;
}

// 1 / prod_{m != b} (b - m)
template <int Q>
__host__ __device__ constexpr double node_scale(int b)
{
  double den = 1.0;
  for(int m = 0; m <= Q; ++m)
    if(m != b) den *= (double)(b - m);
  return 1.0 / den;
}

// FP64 Lagrange weights at fraction x as w0, d1 and s2 with w1 = w0 d1 / dt and
// w2 = w0 s2 / dt^2: d1 = -sum 1/(x-m) and s2 = d1^2 - sum 1/(x-m)^2 over the
// other nodes, added in the reference's order and rounded term by term as it
// rounds them (lagrange_set.cpp:17-41).  Near x = 0 and x = 1 those sums
// cancel and their rounding dominates a pair's error; a form without
// reciprocals is some 500 times more accurate there (rms over random pairs),
// but stands as far from the table's coefficients as those are from the
// exact ones.  Calls tap(b, w0, d1, s2) for b = 0 .. Q; x = 0 gives NaN for
// every node but the first.
template <int Q, class F>
__device__ __forceinline__ void lagrange_taps(double x, const F &tap)
{
  double f[Q + 1], r[Q + 1], sq[Q + 1], above[Q + 1];
#pragma unroll
  for(int m = 0; m <= Q; ++m) {
    f[m] = x - m;
    r[m] = rcp_newton(f[m]);
    sq[m] = r[m] * r[m];
  }
  above[Q] = 1.0;  // prod_{m > b} f_m
#pragma unroll
  for(int b = Q; b > 0; --b) above[b - 1] = above[b] * f[b];
  double below = 1.0, p1 = 0.0, p2 = 0.0;  // over m < b
#pragma unroll
  for(int b = 0; b <= Q; ++b) {
    double d1 = p1, d2 = p2;
#pragma unroll
    for(int m = b + 1; m <= Q; ++m) {
      d1 = d1 - r[m];
      d2 = d2 - sq[m];
    }
    tap(b, (below * above[b]) * node_scale<Q>(b), d1, d2 + d1 * d1);
    below = below * f[b];
    p1 = p1 - r[b];
    p2 = p2 - sq[b];
  }
}

__device__ __forceinline__ void put_tap(double2 &c, double re, double im) { c = make_double2(re, im); }
__device__ __forceinline__ void put_tap(double &c, double re, double) { c = re; }

// One pair's taps (c: complex in the rotating frame, real in
// the lab frame), in an algebraically equal but cheaper form of
// pair_coef_ref.  The dyads are contracted with the dipoles first:
// d_obs.(I - 3 rr).d_src = dd - 3 (d_obs.r)(d_src.r)/r^2 and d_obs.(I - rr).d_src
// = dd - (d_obs.r)(d_src.r)/r^2, so each tap needs three real scalars
//   G0 = (dd - 3ab/r^2) c^2/r^3, G1 = (dd - 3ab/r^2) c/r^2, G2 = (dd - ab/r^2)/r;
//   rotating frame     coef_i = s (G0 w0 + G1 (w1 + i om w0) + G2 (w2 + 2 i om w1
//                      - om^2 w0)), s = -mu0/(4 pi hbar) e^{-i om r/c};
//   lab frame          coef_i = mu0/(4 pi hbar) (G0 w0 + G1 w1 + G2 w2).
// A tap is then alpha w0 + beta w1 + gamma w2 with three factors per pair.
// Every quantity is symmetric in the two dots to the bit, so the pair's
// orientation does not matter.  At an integer delay the reference's weights of
// every node but the first are NaN (lagrange_set.cpp:25-33), and so are the
// taps.
template <int Q, bool LAB, class C>
__device__ __forceinline__ void pair_coef_otf(const PairGeom &g, const double (&da)[3], const double (&db)[3],
                                              const OtfConst &o, C (&c)[Q + 1])
{
  const double dd = fma(da[2], db[2], fma(da[1], db[1], da[0] * db[0]));
  const double ar = fma(da[2], g.dr[2], fma(da[1], g.dr[1], da[0] * g.dr[0]));
  const double br = fma(db[2], g.dr[2], fma(db[1], g.dr[1], db[0] * g.dr[0]));
  const double inv_r = rcp_newton(g.nrm), inv_sq = inv_r * inv_r;
  const double ab = (ar * br) * inv_sq;
  const double g3 = fma(-3.0, ab, dd), g1 = dd - ab;
  const double G2 = g1 * inv_r, G1 = (g3 * o.c0) * inv_sq, G0 = (g3 * o.c0_sq) * (inv_sq * inv_r);
  if(LAB) {
    const double al = o.A * G0, be = (o.A * G1) * o.inv_dt, ga = (o.A * G2) * o.inv_dt2;
    lagrange_taps<Q>(g.x, [&](int b, double w0, double d1, double s2) {
      put_tap(c[b], w0 * fma(ga, s2, fma(be, d1, al)), 0.0);
    });
  } else {
    double sn, cs;
    sincospi(half_turns(g.nrm, o), &sn, &cs);
    const double sx = -(o.A * cs), sy = o.A * sn;  // s = -A e^{-i omega r / c0}
    const double ar0 = fma(-o.om_sq, G2, G0), ai0 = o.om * G1;
    const double br0 = G1 * o.inv_dt, bi0 = 2.0 * (o.om * G2) * o.inv_dt;
    const double gr0 = G2 * o.inv_dt2;
    const double alx = fma(sx, ar0, -(sy * ai0)), aly = fma(sx, ai0, sy * ar0);
    const double bex = fma(sx, br0, -(sy * bi0)), bey = fma(sx, bi0, sy * br0);
    const double gax = sx * gr0, gay = sy * gr0;
    lagrange_taps<Q>(g.x, [&](int b, double w0, double d1, double s2) {
      put_tap(c[b], w0 * fma(gax, s2, fma(bex, d1, alx)), w0 * fma(gay, s2, fma(bey, d1, aly)));
    });
  }
}

// Lagrange node products with their first two derivatives: with
// f_m = x - m, value = prod f_m, d1 = its derivative, h2 = half its second
// derivative.  A node's weights (lagrange_set.cpp:17-41) leave its own factor
// out: w0 = value / den, w1 = -d1 / (den dt), w2 = 2 h2 / (den dt^2), den =
// prod (b - m).  Taken from the products of the factors below and above the
// node, without reciprocals (whose 1/x-sized terms cancel as x -> 0) and at
// six operations a node.
template <class T>
struct Jet {
  T v, d, h;
  // times the factor f = x - m
  __device__ __forceinline__ Jet times(T f) const
  {
    Jet r;
    r.v = v * f;
    r.d = fma_(d, f, v);
    r.h = fma_(h, f, d);
    return r;
  }
  __device__ __forceinline__ Jet times(const Jet &o) const
  {
    Jet r;
    r.v = v * o.v;
    r.d = fma_(d, o.v, v * o.d);
    r.h = fma_(h, o.v, fma_(d, o.d, v * o.h));
    return r;
  }
  static __device__ __forceinline__ double fma_(double a, double b, double c) { return fma(a, b, c); }
  static __device__ __forceinline__ float fma_(float a, float b, float c) { return fmaf(a, b, c); }
};

// calls tap(b, jet) for b = Q .. 0
template <int Q, class T, class F>
__device__ __forceinline__ void lagrange_jets(T x, const F &tap)
{
  Jet<T> below[Q + 1];  // prod_{m < b}
  below[0] = Jet<T>{T(1), T(0), T(0)};
#pragma unroll
  for(int b = 0; b < Q; ++b)
    below[b + 1] = b == 0 ? Jet<T>{x, T(1), T(0)} : below[b].times(x - T(b));
  Jet<T> above{T(1), T(0), T(0)};  // prod_{m > b}
#pragma unroll
  for(int b = Q; b >= 0; --b) {
    tap(b, b == Q ? below[b] : b == 0 ? above : below[b].times(above));
    if(b > 0) above = b == Q ? Jet<T>{x - T(b), T(1), T(0)} : above.times(x - T(b));
  }
}

// Mixed-precision taps of one pair.  FP64 is kept for the distance and the
// split of r / (c dt) into the floor delay and the fraction, for 1/r, and for
// reducing the phase omega r / c to one turn; the Lagrange weights, the dyad
// factors and the taps are FP32.
//
// cf[0..Q] are the taps and cf[Q+1] their sum, taken from the identities
// sum w0 = 1, sum w1 = sum w2 = 0 as the w0-only coefficient: the
// difference-form convolution multiplies the sum by the window's first
// sample and each tap by a step difference, so the sum must be accurate to
// FP32 rounding while the taps (each ~1e-7 relative) only meet differences.
// An integer delay (x = 0) gives NaN taps 1..Q (and sum) and a finite tap 0,
// as the reference's weights do, so a run turns non-finite at the same step.
template <int Q, bool LAB>
__device__ __forceinline__ void pair_coef_otf_mixed(const PairGeom &g, const double (&da)[3], const double (&db)[3],
                                                    const OtfConst &o, float2 (&cf)[Q + 2])
{
  const float x = (float)g.x;
  const float drf[3] = {(float)g.dr[0], (float)g.dr[1], (float)g.dr[2]};
  const float fa[3] = {(float)da[0], (float)da[1], (float)da[2]};
  const float fb[3] = {(float)db[0], (float)db[1], (float)db[2]};
  const float dd = fmaf(fa[2], fb[2], fmaf(fa[1], fb[1], fa[0] * fb[0]));
  const float ar = fmaf(fa[2], drf[2], fmaf(fa[1], drf[1], fa[0] * drf[0]));
  const float br = fmaf(fb[2], drf[2], fmaf(fb[1], drf[1], fb[0] * drf[0]));
  const float inv_r = (float)rcp_newton(g.nrm), inv_sq = inv_r * inv_r;
  const float ab = (ar * br) * inv_sq;
  const float g3 = fmaf(-3.f, ab, dd), g1 = dd - ab;
  const float G0 = (g3 * (float)o.c0_sq) * (inv_sq * inv_r);
  const float G1 = (g3 * (float)o.c0) * inv_sq;
  const float G2 = g1 * inv_r;
  const float A = (float)o.A, idt = (float)o.inv_dt, idt2 = (float)(2.0 * o.inv_dt2);
  if(LAB) {
    const float al = A * G0, be = -(A * G1) * idt, ga = (A * G2) * idt2;
    lagrange_jets<Q>(x, [&](int b, const Jet<float> &j) {
      cf[b] = make_float2((float)node_scale<Q>(b) * fmaf(ga, j.h, fmaf(be, j.d, al * j.v)), 0.f);
    });
    cf[Q + 1] = make_float2(al, 0.f);
  } else {
    const double ph = g.nrm * o.half_turns;
    float sn, cs;
    sincospif((float)fma(-2.0, rint(0.5 * ph), ph), &sn, &cs);
    const float sx = -(A * cs), sy = A * sn;
    const float om = (float)o.om;
    const float ar0 = fmaf(-(float)o.om_sq, G2, G0), ai0 = om * G1;
    const float br0 = -G1 * idt, bi0 = -2.f * (om * G2) * idt;
    const float gr0 = G2 * idt2;
    const float alx = fmaf(sx, ar0, -(sy * ai0)), aly = fmaf(sx, ai0, sy * ar0);
    const float bex = fmaf(sx, br0, -(sy * bi0)), bey = fmaf(sx, bi0, sy * br0);
    const float gax = sx * gr0, gay = sy * gr0;
    lagrange_jets<Q>(x, [&](int b, const Jet<float> &j) {
      const float id = (float)node_scale<Q>(b);
      cf[b] = make_float2(id * fmaf(gax, j.h, fmaf(bex, j.d, alx * j.v)), id * fmaf(gay, j.h, fmaf(bey, j.d, aly * j.v)));
    });
    cf[Q + 1] = make_float2(alx, aly);
  }
  if(g.x == 0.0) {
#pragma unroll
    for(int i = 1; i <= Q + 1; ++i) cf[i] = make_float2(__int_as_float(0x7fc00000), 0.f);
  }
}

}  // namespace qg
