// Convolution and reduction pieces shared by the far-pair kernels (table
// and on-the-fly coefficients).  Every product is an explicit fused
// multiply-add and every other operation a plain add, so the results do not
// depend on the translation unit's contraction setting.
#pragma once

#include <cuda_runtime.h>

#include "qg_internal.h"

namespace qg {

// ---- accumulators --------------------------------------------------------------
// One lane's K far-field sums.  Rotating frame: complex taps on complex
// samples.  Lab frame (prefactor 2 Re rho01, real taps): real products only.
// The imaginary part of a complex product of them is zero, or NaN where a
// factor is not finite (and the real part is not either): v * 0.
template <bool LAB, int K>
struct FarAcc;

template <int K>
struct FarAcc<false, K> {
  using C = double2;
  double2 v[K];
  __device__ __forceinline__ void zero()
  {
#pragma unroll
    for(int k = 0; k < K; ++k) v[k] = make_double2(0.0, 0.0);
  }
  static __device__ __forceinline__ C load(const double2 *p) { return __ldcs(p); }
  static __device__ __forceinline__ C from(double2 c) { return c; }
  // sample m's products with the taps of the outputs it feeds: the two
  // multiply-adds of a sum are dependent, so the first of every sum come
  // before the second of any
  template <int Q>
  __device__ __forceinline__ void sample(int m, const C (&c)[Q + 1], double2 r)
  {
#pragma unroll
    for(int k = (m - Q > 0 ? m - Q : 0); k <= (m < K - 1 ? m : K - 1); ++k) {
      v[k].x = fma(c[k + Q - m].x, r.x, v[k].x);
      v[k].y = fma(c[k + Q - m].x, r.y, v[k].y);
    }
#pragma unroll
    for(int k = (m - Q > 0 ? m - Q : 0); k <= (m < K - 1 ? m : K - 1); ++k) {
      v[k].x = fma(-c[k + Q - m].y, r.y, v[k].x);
      v[k].y = fma(c[k + Q - m].y, r.x, v[k].y);
    }
  }
  __device__ __forceinline__ double2 out(int k) const { return v[k]; }
};

template <int K>
struct FarAcc<true, K> {
  using C = double;
  double v[K];
  __device__ __forceinline__ void zero()
  {
#pragma unroll
    for(int k = 0; k < K; ++k) v[k] = 0.0;
  }
  static __device__ __forceinline__ C load(const double2 *p) { return __ldcs(&p->x); }
  static __device__ __forceinline__ C from(double2 c) { return c.x; }
  template <int Q>
  __device__ __forceinline__ void sample(int m, const C (&c)[Q + 1], double2 r)
  {
    const double x = 2 * r.x;
#pragma unroll
    for(int k = (m - Q > 0 ? m - Q : 0); k <= (m < K - 1 ? m : K - 1); ++k) v[k] = fma(c[k + Q - m], x, v[k]);
  }
  __device__ __forceinline__ double2 out(int k) const { return make_double2(v[k], v[k] * 0.0); }
};

// Packed FP32 pairs (Blackwell fma.rn.f32x2 / add.rn.f32x2): one instruction
// does two independent FP32 operations, each rounded as the scalar one is.
__device__ __forceinline__ unsigned long long pk2(float2 v)
{
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(v.x), "f"(v.y));
  return r;
}
__device__ __forceinline__ float2 upk2(unsigned long long r)
{
  float2 v;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(r));
  return v;
}
__device__ __forceinline__ unsigned long long ffma2(unsigned long long a, unsigned long long b, unsigned long long c)
{
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long fadd2(unsigned long long a, unsigned long long b)
{
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// Accumulators of the mixed-precision convolution (difference form, see
// qg_far.cu).  A complex multiply-add acc += c u is kept as two real pairs,
// a += (c.x, c.x) (u.x, u.y) and b += (c.y, c.y) (u.x, u.y), so a packed
// FP32 pair instruction (fma.rn.f32x2) does each without first swapping u's
// halves; the product's real part is a.x - b.y and its imaginary part
// a.y + b.x, formed in FP64 when the partial is written.  `base` collects the
// tap-sum term (sum_i c_i) w_0, which is the same for all K outputs of a
// pair, once per pair.  The lab frame's taps and samples are real: one
// scalar multiply-add each.
template <bool LAB, int Q, int K>
struct MixedAcc;

template <int Q, int K>
struct MixedAcc<false, Q, K> {
  unsigned long long a[K], b[K];
  float2 base;
  unsigned long long cx[Q + 1], cy[Q + 1];  // the current pair's taps
  unsigned long long u;                     // its running sum of differences
  __device__ __forceinline__ void zero()
  {
#pragma unroll
    for(int k = 0; k < K; ++k) a[k] = b[k] = pk2(make_float2(0.f, 0.f));
    base = make_float2(0.f, 0.f);
  }
  __device__ __forceinline__ void taps(const float2 (&c)[Q + 2])
  {
#pragma unroll
    for(int i = 0; i <= Q; ++i) {
      cx[i] = pk2(make_float2(c[i].x, c[i].x));
      cy[i] = pk2(make_float2(c[i].y, c[i].y));
    }
    u = pk2(make_float2(0.f, 0.f));
  }
  __device__ __forceinline__ void first(float2 csum, float2 w0)
  {
    base.x = fmaf(csum.x, w0.x, base.x);
    base.x = fmaf(-csum.y, w0.y, base.x);
    base.y = fmaf(csum.x, w0.y, base.y);
    base.y = fmaf(csum.y, w0.x, base.y);
  }
  __device__ __forceinline__ void add(float2 d) { u = fadd2(u, pk2(d)); }
  // the skipping loop's absolute sample w_0 + u
  __device__ __forceinline__ unsigned long long absolute(float2 w0) const
  {
    const float2 v = upk2(u);
    return pk2(make_float2(w0.x + v.x, w0.y + v.y));
  }
  __device__ __forceinline__ void mac(int k, int i, unsigned long long w)
  {
    a[k] = ffma2(cx[i], w, a[k]);
    b[k] = ffma2(cy[i], w, b[k]);
  }
  __device__ __forceinline__ double2 out(int k) const
  {
    const float2 p = upk2(a[k]), r = upk2(b[k]);
    return make_double2(((double)p.x - (double)r.y) + (double)base.x, ((double)p.y + (double)r.x) + (double)base.y);
  }
};

template <int Q, int K>
struct MixedAcc<true, Q, K> {
  float a[K];
  float base;
  float cx[Q + 1];
  float u;
  __device__ __forceinline__ void zero()
  {
#pragma unroll
    for(int k = 0; k < K; ++k) a[k] = 0.f;
    base = 0.f;
  }
  __device__ __forceinline__ void taps(const float2 (&c)[Q + 2])
  {
#pragma unroll
    for(int i = 0; i <= Q; ++i) cx[i] = c[i].x;
    u = 0.f;
  }
  __device__ __forceinline__ void first(float2 csum, float2 w0) { base = fmaf(csum.x, 2.f * w0.x, base); }
  __device__ __forceinline__ void add(float2 d) { u += 2.f * d.x; }
  __device__ __forceinline__ float absolute(float2 w0) const { return 2.f * w0.x + u; }
  __device__ __forceinline__ void mac(int k, int i, float w) { a[k] = fmaf(cx[i], w, a[k]); }
  __device__ __forceinline__ double2 out(int k) const
  {
    const double v = (double)a[k] + (double)base;
    return make_double2(v, v * 0.0);
  }
};

// ---- windows read from the ring ------------------------------------------------
// acc[k] += sum_i c[i] * w[k + Q - i] over the window w[m] = ring[slot0 + m],
// m = 0 .. K+Q-1, whose first sample is step tau0.  Samples before step -22
// are skipped (their taps are skipped by the reference; kFormPlain: none need
// be): a warp with such a sample takes the second loop for all its lanes,
// whose reads do not wait for the tests (every sample of a window lies in the
// ring row).
template <int Q, bool LAB, int K, int FORM>
__device__ __forceinline__ void window_conv(const double2 *ring, int slot0, int tau0,
                                            const typename FarAcc<LAB, K>::C (&c)[Q + 1], FarAcc<LAB, K> &acc)
{
  if(FORM == kFormPlain || __all_sync(__activemask(), tau0 >= -kWindow)) {
#pragma unroll
    for(int m = 0; m < K + Q; ++m) acc.template sample<Q>(m, c, __ldg(ring + slot0 + m));
  } else {
#pragma unroll
    for(int m = 0; m < K + Q; ++m) {
      const double2 w = __ldg(ring + slot0 + m);
      if(tau0 + m >= -kWindow) acc.template sample<Q>(m, c, w);
    }
  }
}

// acc[k] += sum_i c_i w_{k+Q-i} over the window w_m, m = 0 .. K+Q-1, whose
// first sample w_0 (step tau0) is rw[slot0] and whose later samples are
// w_0 + u_m, u_m the running sum of the FP32 step-to-step differences
// rd[slot0 + 1 .. slot0 + m].  c[Q+1] is the pair's tap sum.  When every
// sample is live (tau0 >= -22) this is (sum_i c_i) w_0 + sum_i c_i u_{k+Q-i}:
// the first term goes to `base` once and the differences meet only the taps.
// Samples before step -22 are skipped (their taps are skipped by the
// reference); there the absolute samples w_0 + u_m meet the live taps.
template <int Q, bool LAB, int K, int FORM>
__device__ __forceinline__ void window_conv_mixed(const float2 *rw, const float2 *rd, int slot0, int tau0,
                                                  const float2 (&c)[Q + 2], MixedAcc<LAB, Q, K> &acc)
{
  const float2 w0 = __ldg(rw + slot0);
  acc.taps(c);
  if(FORM == kFormPlain || tau0 >= -kWindow) {
    acc.first(c[Q + 1], w0);
#pragma unroll
    for(int m = 1; m < K + Q; ++m) {
      acc.add(__ldg(rd + slot0 + m));
#pragma unroll
      for(int k = (m - Q > 0 ? m - Q : 0); k <= (m < K - 1 ? m : K - 1); ++k) acc.mac(k, k + Q - m, acc.u);
    }
  } else {
#pragma unroll
    for(int m = 0; m < K + Q; ++m) {
      if(m > 0) acc.add(__ldg(rd + slot0 + m));
      if(tau0 + m < -kWindow) continue;
      const auto w = acc.absolute(w0);
#pragma unroll
      for(int k = (m - Q > 0 ? m - Q : 0); k <= (m < K - 1 ? m : K - 1); ++k) acc.mac(k, k + Q - m, w);
    }
  }
}

// ---- tasks and partials ------------------------------------------------------------
__device__ __forceinline__ int wrap_slot(int t, int W)
{
  const int s = t % W;
  return s < 0 ? s + W : s;
}

// A warp's task: one target tile and the sources [s0, s1) of one part (s1 <=
// s0: an empty part).  Neighbouring tasks, the warps of a block, share the
// part's sources, so they read the same history rows.
struct FarTask {
  int I, part, s0, s1;
};
__device__ __forceinline__ FarTask far_task(const FarArgs &a, int task)
{
  const int tiles = a.tile_n > 0 ? a.tile_n : a.nT;
  FarTask t;
  t.part = task / tiles;
  t.I = a.tile_lo + task - t.part * tiles;
  const int g = t.part / a.parts, j = t.part - g * a.parts;
  t.s0 = g * a.group * kTile + j * a.unit;
  t.s1 = min(t.s0 + a.unit, min((g + 1) * a.group, a.nT) * kTile);
  return t;
}

// A lane's K sums as its target's partial of the part.
template <int K, class Acc>
__device__ __forceinline__ void store_partial(const FarArgs &a, const FarTask &t, const Acc &acc)
{
  const long long slice = (long long)a.nP * a.n_pad;
  double2 *out = a.partial + (long long)t.part * a.n_pad + t.I * kTile + (threadIdx.x & 31);
#pragma unroll
  for(int k = 0; k < K; ++k) out[k * slice] = acc.out(k);
}

}  // namespace qg
