// Far-pair kernel with on-the-fly coefficients: the same K-step sum as the
// table path (qg_far.cu) for ensembles whose coefficient table does not fit
// in device memory (N = 65536 needs 215 GB in FP64).  Each warp owns a target
// tile (lane = target dot) and one part of the sources; for every source the
// 32 lanes compute their pair's floor delay and q+1 coefficients
// (pair_coef_otf) and, for pairs with delay >= K, apply them to the source's
// K + q window exactly as the table path does.  The coefficients are computed
// once per pair per K steps.
//
// FP64: FP64 coefficients and convolution.  Mixed: FP32 coefficients
// (pair_coef_otf_mixed: FP64 only for the distance, the delay split and the
// phase reduction) with their sum from the Lagrange identities, and the FP32
// difference-form convolution of the mixed table path.
//
// Compiled with -fmad=false (the delay arithmetic must match the near-pair
// search bit for bit); the convolution's products are explicit fused
// multiply-adds, so they round as in the table path.
#include <cuda_runtime.h>

#include "qg_coef.cuh"
#include "qg_conv.cuh"

namespace qg {

// One pair's taps and its window's convolution.
template <int Q, bool LAB, bool MIXED, int K, int FORM>
struct OtfPair;

template <int Q, bool LAB, int K, int FORM>
struct OtfPair<Q, LAB, false, K, FORM> {
  using Acc = FarAcc<LAB, K>;
  typename Acc::C c[Q + 1];
  __device__ __forceinline__ void make(const PairGeom &g, const double (&da)[3], const double (&db)[3],
                                       const OtfConst &oc)
  {
    pair_coef_otf<Q, LAB>(g, da, db, oc, c);
  }
  __device__ __forceinline__ void conv(const FarArgs &a, int ib, int tau0, Acc &acc) const
  {
    window_conv<Q, LAB, K, FORM>(a.ring + (long long)ib * a.stride, wrap_slot(tau0, a.W), tau0, c, acc);
  }
};

template <int Q, bool LAB, int K, int FORM>
struct OtfPair<Q, LAB, true, K, FORM> {
  using Acc = MixedAcc<LAB, Q, K>;
  float2 c[Q + 2];
  __device__ __forceinline__ void make(const PairGeom &g, const double (&da)[3], const double (&db)[3],
                                       const OtfConst &oc)
  {
    pair_coef_otf_mixed<Q, LAB>(g, da, db, oc, c);
  }
  __device__ __forceinline__ void conv(const FarArgs &a, int ib, int tau0, Acc &acc) const
  {
    window_conv_mixed<Q, LAB, K, FORM>(a.ring32w + (long long)ib * a.stride, a.ring32d + (long long)ib * a.stride,
                                 wrap_slot(tau0, a.W), tau0, c, acc);
  }
};

// K steps (the run's far kernel) or one (evaluations).  Held to 3 blocks on
// an SM (168 registers).
template <int Q, bool LAB, bool MIXED, int K, int FORM>
__global__ void __launch_bounds__(32 * kFarWarps, 3) far_otf_kernel(FarArgs a)
{
  using Pair = OtfPair<Q, LAB, MIXED, K, FORM>;
  const int lane = threadIdx.x & 31;
  const int task = blockIdx.x * kFarWarps + (threadIdx.x >> 5);
  const int t0 = *a.d_t0;
  if(blockIdx.x == 0 && threadIdx.x == 0) *a.far_t0_out = t0;
  if(task >= far_tasks(a)) return;  // uniform per warp
  const FarTask t = far_task(a, task);
  // a window of delay d has a sample at step -22 or later
  const int d_last = t0 + K - 1 + kWindow;
  const int ia = t.I * kTile + lane;
  const bool target = a.user[ia] >= 0;
  const double pa[3] = {a.pos[3 * ia], a.pos[3 * ia + 1], a.pos[3 * ia + 2]};
  const double da[3] = {a.dip[3 * ia], a.dip[3 * ia + 1], a.dip[3 * ia + 2]};
  typename Pair::Acc acc;
  acc.zero();
#pragma unroll 1
  for(int s = t.s0; s < t.s1; ++s) {
    if(__ldg(a.user + s) < 0) continue;  // the same source for all lanes
    const double pb[3] = {__ldg(a.pos + 3 * s), __ldg(a.pos + 3 * s + 1), __ldg(a.pos + 3 * s + 2)};
    const PairGeom g = pair_geom(pa, pb, a.oc);
    const bool live = target && ia != s && g.fd >= kTimeBlock && g.fd <= d_last;
    if(!__any_sync(0xffffffffu, live)) continue;
    const double db[3] = {__ldg(a.dip + 3 * s), __ldg(a.dip + 3 * s + 1), __ldg(a.dip + 3 * s + 2)};
    Pair pair;
    pair.make(g, da, db, a.oc);
    if(live) pair.conv(a, s, t0 - g.fd - Q, acc);
    __syncwarp();
  }
  store_partial<K>(a, t, acc);
}

template <bool LAB, bool MIXED, int K, int FORM>
static void launch_otf_frame(const FarArgs &a, cudaStream_t s)
{
#define QG_OTF_CASE(QQ) \
  case QQ: far_otf_kernel<QQ, LAB, MIXED, K, FORM><<<far_blocks(a), 32 * kFarWarps, 0, s>>>(a); break;
  switch(a.q) {
    QG_OTF_CASE(1)
    QG_OTF_CASE(2)
    QG_OTF_CASE(3)
    QG_OTF_CASE(4)
    QG_OTF_CASE(5)
    QG_OTF_CASE(6)
    QG_OTF_CASE(7)
    default: break;
  }
#undef QG_OTF_CASE
}

template <int K, int FORM>
static void launch_otf(const FarArgs &a, cudaStream_t s)
{
  if(a.nT <= 0) return;
  if(a.frame == 0)
    a.mixed ? launch_otf_frame<false, true, K, FORM>(a, s) : launch_otf_frame<false, false, K, FORM>(a, s);
  else
    a.mixed ? launch_otf_frame<true, true, K, FORM>(a, s) : launch_otf_frame<true, false, K, FORM>(a, s);
}

void launch_far_otf(const FarArgs &a, void *stream)
{
  if(a.form == kFormPlain)
    launch_otf<kTimeBlock, kFormPlain>(a, (cudaStream_t)stream);
  else
    launch_otf<kTimeBlock, kFormAny>(a, (cudaStream_t)stream);
}
void launch_far_otf_step1(const FarArgs &a, void *stream) { launch_otf<1, kFormAny>(a, (cudaStream_t)stream); }

}  // namespace qg
