// Far-pair kernel: K = kTimeBlock steps of the retarded pair sum from one
// pass over the coefficient table.
//
// HistoryInteraction::evaluate (reference history_interaction.cpp:47-70)
// sums, for every unordered pair (a, b) and tap i = 0..q,
//     field[a] += prefactor(rho01_b[s-i]) * coef_i,
//     field[b] += prefactor(rho01_a[s-i]) * coef_i,   s = step - delay_ab,
// skipping taps with s - i < -22, and the integrator calls it 11 times per
// step (integrator.cpp:133-139).  For a pair with floor delay d >= K every
// tap of every step in [t0, t0 + K) reads a step before t0, so its K x (q+1)
// terms are fixed once step t0 - 1 is done: one pass over the table at t0
// gives the far-pair part of the field for the next K steps.  Pairs with
// d < K (a few per thousand at the benchmark sizes) are summed per step by
// the dot-step kernel from a compact list.
//
// Per ordered pair the K steps read one window of K + q consecutive history
// samples of the source and form a K-output, (q+1)-tap convolution with the
// pair's coefficients: K (q+1) complex multiply-adds per ordered pair per
// pass, each coefficient read from HBM once per K steps.  The window is
// consumed one sample at a time (each sample feeds up to q+1 outputs), so
// only the K accumulators and the q+1 coefficients stay in registers.
//
// Schedule.  One warp owns a target tile I (lane l = dot 32 I + l) and one
// part of the sources.  At each step all 32 lanes take the same source b, so
// their windows, at the 32 different delays d(a_l, b), fall in one short
// stretch of b's history row: a handful of cache lines per load instead of
// 32.  The table's entries are copied asynchronously into the warp's own
// shared memory (FP64) or prefetched in registers (mixed), a source ahead, the
// delays earlier still.  A warp none of whose windows
// reaches step -22 yet skips the source, its coefficients included, so the
// first blocks of a run cost what they use.
//
// Each part's sums go to a partial and a second launch adds the partials in
// part order, so the result does not depend on scheduling.
//
// The rho01 ring holds rho01 by time slot (slot = t mod W) with the first
// kRingMirror slots repeated after slot W-1, so every window is contiguous.
// Polarisation prefactor: rho01 in the rotating frame
// (rotating_green_function.h:17-21), 2 Re rho01 in the lab frame
// (green_function.h:23-27).
//
// Mixed precision.  The tap sum of one pair, sum_i c_i w_i, is formed as
//     (sum_i c_i) w_0 + sum_i c_i (w_i - w_0),
// w_0 the window's first sample and w_i - w_0 the running sum of the FP32
// step-to-step differences (themselves computed in FP64).  The large
// interpolation weights (w1 ~ 1/dt, w2 ~ 1/dt^2) multiply only differences,
// and sum_i c_i carries no such factor, so FP32 storage loses no more than a
// few units in the last place of the pair's contribution.  The first term is
// the same for all K outputs and is accumulated once per pair (MixedAcc).
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <type_traits>

#include "qg_conv.cuh"

namespace qg {

// Three blocks of 4 warps on an SM (168 registers) for FP64, four (128) for
// the mixed form.
template <bool MIXED>
constexpr int kFarBlocks = MIXED ? 4 : 3;

// FP64: each lane copies its own entries of the table into its warp's shared
// memory: a source's q+1 coefficients one source ahead (evict-first in L2: the
// table is streamed once per launch, the history ring should stay), its delay
// kDelayAhead sources ahead.  Delays prefetched in registers are moved from
// one to the next on every source, and the move waits for the load: a source
// that every window skips cost 0.9 us.  First block of 4096 dots 284 -> 252 us,
// a steady launch 642 -> 632 us, of 1500 dots 114 -> 111 us.  Coefficients two
// sources ahead leave less to L1: 642 instead of 627 us at 4096 dots.
constexpr int kDelayAhead = 4;
constexpr int kDelaySlots = 8;

template <int Q>
struct FarStage {
  double2 coef[2][Q + 1][32];
  int delay[kDelaySlots][32];
};

__device__ __forceinline__ void cp_async16(void *dst, const void *src, unsigned long long pol)
{
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "l"(pol) : "memory");
}
__device__ __forceinline__ void cp_async4(void *dst, const void *src, unsigned long long pol)
{
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global.L2::cache_hint [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "l"(pol) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait()
{
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

template <int Q, bool LAB, bool MIXED, int FORM>
struct FarBody;

// Each lane reads back only what it copied.  One group of copies per source:
// group s holds the coefficients of source s + 1 and the delays of source
// s + kDelayAhead, so with all but the newest kDelayAhead - 2 groups done the
// delays of source s + 1 are there, and with all but the newest one the
// coefficients of source s.
template <int Q, bool LAB, int FORM>
struct FarBody<Q, LAB, false, FORM> {
  using Shared = FarStage<Q>;
  static __device__ __forceinline__ void run(const FarArgs &a, const FarTask &t, int t0, Shared &st)
  {
    constexpr int K = kTimeBlock;
    static_assert(kDelayAhead > 2 && kDelaySlots > kDelayAhead, "a slot is read before it is copied to again");
    using Acc = FarAcc<LAB, K>;
    const int lane = threadIdx.x & 31;
    // a window of delay d has a sample at step -22 or later
    const int d_last = t0 + K - 1 + kWindow;
    unsigned long long pol;
    asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
    const long long tile = (long long)t.I * a.nT;
    // a tile row's delays are one array over the sources, 32 entries each
    const int *dp = a.delay + tile * kTilePairs + lane;
    auto fetch_delay = [&](int s) {
      if(s < t.s1) cp_async4(&st.delay[s % kDelaySlots][lane], dp + s * kTile, pol);
    };
    // the delay of source s, -1 where no window is to be read
    auto delay = [&](int s) {
      if(s >= t.s1) return -1;
      const int d = st.delay[s % kDelaySlots][lane];
      return d >= K && d <= d_last ? d : -1;
    };
    auto fetch_coef = [&](int s, int d) {
      if(!__any_sync(0xffffffffu, d >= 0)) return;
      const double2 *src = a.coef + ((tile + s / kTile) * (Q + 1)) * kTilePairs + (s % kTile) * kTile + lane;
#pragma unroll
      for(int i = 0; i <= Q; ++i) cp_async16(&st.coef[s & 1][i][lane], src + i * kTilePairs, pol);
    };
    Acc acc;
    acc.zero();
#pragma unroll
    for(int s = 0; s < kDelayAhead; ++s) fetch_delay(t.s0 + s);
    cp_async_commit();
    cp_async_wait<0>();
    int d0 = delay(t.s0);
    fetch_coef(t.s0, d0);
    cp_async_commit();
#pragma unroll 1
    for(int s = t.s0; s < t.s1; ++s) {
      cp_async_wait<kDelayAhead - 2>();
      const int d1 = delay(s + 1);
      fetch_coef(s + 1, d1);
      fetch_delay(s + kDelayAhead);
      cp_async_commit();
      cp_async_wait<1>();
      if(d0 >= 0) {
        typename Acc::C c[Q + 1];
#pragma unroll
        for(int i = 0; i <= Q; ++i) c[i] = Acc::from(st.coef[s & 1][i][lane]);
        const int tau0 = t0 - d0 - Q;
        window_conv<Q, LAB, K, FORM>(a.ring + (long long)s * a.stride, wrap_slot(tau0, a.W), tau0, c, acc);
      }
      __syncwarp();
      d0 = d1;
    }
    cp_async_wait<0>();
    store_partial<K>(a, t, acc);
  }
};

template <int Q, bool LAB, int FORM>
struct FarBody<Q, LAB, true, FORM> {
  struct Shared {
  };
  static __device__ __forceinline__ void run(const FarArgs &a, const FarTask &t, int t0, Shared &)
  {
    constexpr int K = kTimeBlock;
    const int lane = threadIdx.x & 31;
    const int d_last = t0 + K - 1 + kWindow;
    const long long tile = (long long)t.I * a.nT;
    const int *dp = a.delay + tile * kTilePairs + lane;
    auto load_delay = [&](int s) { return s < t.s1 ? __ldcs(dp + s * kTile) : -1; };
    auto live = [&](int d) { return d >= K && d <= d_last; };
    float2 next[Q + 2];
    auto load = [&](int s, int d) {
      if(__any_sync(0xffffffffu, live(d))) {
        const float2 *src = a.coef32 + ((tile + s / kTile) * (Q + 2)) * kTilePairs + (s % kTile) * kTile + lane;
#pragma unroll
        for(int i = 0; i <= Q + 1; ++i) next[i] = __ldcs(src + i * kTilePairs);
      }
    };
    MixedAcc<LAB, Q, K> acc;
    acc.zero();
    int d0 = load_delay(t.s0), d1 = load_delay(t.s0 + 1);
    load(t.s0, d0);
#pragma unroll 1
    for(int s = t.s0; s < t.s1; ++s) {
      float2 c[Q + 2];
#pragma unroll
      for(int i = 0; i <= Q + 1; ++i) c[i] = next[i];
      load(s + 1, d1);
      const int d2 = load_delay(s + 2);
      if(live(d0)) {
        const int tau0 = t0 - d0 - Q;
        window_conv_mixed<Q, LAB, K, FORM>(a.ring32w + (long long)s * a.stride, a.ring32d + (long long)s * a.stride,
                                     wrap_slot(tau0, a.W), tau0, c, acc);
      }
      __syncwarp();
      d0 = d1, d1 = d2;
    }
    store_partial<K>(a, t, acc);
  }
};

template <int Q, bool LAB, bool MIXED, int FORM>
__global__ void __launch_bounds__(32 * kFarWarps, kFarBlocks<MIXED>) far_kernel(FarArgs a)
{
  extern __shared__ __align__(16) char far_smem[];
  using Body = FarBody<Q, LAB, MIXED, FORM>;
  const int w = threadIdx.x >> 5, task = blockIdx.x * kFarWarps + w;
  const int t0 = *a.d_t0;
  if(blockIdx.x == 0 && threadIdx.x == 0) *a.far_t0_out = t0;
  if(task < far_tasks(a)) Body::run(a, far_task(a, task), t0, reinterpret_cast<typename Body::Shared *>(far_smem)[w]);
}

// Many ensembles in one launch: task_off[e] = first block of ensemble e
// (prefix sums).  Every task writes its own partials, so a member's result
// is the one it has alone.
template <int Q, bool LAB, bool MIXED, int FORM>
__global__ void __launch_bounds__(32 * kFarWarps, kFarBlocks<MIXED>)
    far_batch_kernel(const FarArgs *__restrict__ args, const int *__restrict__ task_off, int n_ens)
{
  extern __shared__ __align__(16) char far_smem[];
  using Body = FarBody<Q, LAB, MIXED, FORM>;
  int lo = 0, hi = n_ens - 1;
  while(lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if(task_off[mid] <= (int)blockIdx.x)
      lo = mid;
    else
      hi = mid - 1;
  }
  const FarArgs a = args[lo];  // a copy: the body reads its fields in its loop
  const int blk = blockIdx.x - task_off[lo], w = threadIdx.x >> 5, task = blk * kFarWarps + w;
  const int t0 = *a.d_t0;
  if(blk == 0 && threadIdx.x == 0) *a.far_t0_out = t0;
  if(task < far_tasks(a)) Body::run(a, far_task(a, task), t0, reinterpret_cast<typename Body::Shared *>(far_smem)[w]);
}

// ---- partials --------------------------------------------------------------------
// field[k] of one 32-dot tile: the partials added in part order.
__device__ __forceinline__ void reduce_tile(const FarArgs &a, int tile, int k)
{
  const long long slice = (long long)a.nP * a.n_pad;
  const int ia = tile * kTile + (threadIdx.x & 31);
  const double2 *P = a.partial + k * slice + ia;
  double2 f = make_double2(0.0, 0.0);
#pragma unroll 8
  for(int p = 0; p < a.nP; ++p) {
    const double2 v = __ldcg(P + (long long)p * a.n_pad);
    f.x += v.x;
    f.y += v.y;
  }
  a.field[(long long)k * a.n_pad + ia] = f;
}

__global__ void far_reduce_kernel(FarArgs a) { reduce_tile(a, a.tile_lo + blockIdx.x, threadIdx.x >> 5); }

__global__ void far_reduce_batch_kernel(const FarArgs *__restrict__ args, const int *__restrict__ tile_off, int n_ens)
{
  int lo = 0, hi = n_ens - 1;
  while(lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if(tile_off[mid] <= (int)blockIdx.x)
      lo = mid;
    else
      hi = mid - 1;
  }
  const FarArgs &a = args[lo];
  reduce_tile(a, blockIdx.x - tile_off[lo], threadIdx.x >> 5);
}

void launch_far_reduce(const FarArgs &a, int steps, void *stream)
{
  far_reduce_kernel<<<a.tile_n > 0 ? a.tile_n : a.nT, 32 * steps, 0, (cudaStream_t)stream>>>(a);
}

// ---- launches ----------------------------------------------------------------------
template <int Q, bool MIXED>
constexpr size_t far_smem_bytes()
{
  return MIXED ? 0 : kFarWarps * sizeof(FarStage<Q>);
}
// 28 KB a block at q = 5, 36 KB at the largest order: no opt-in needed
static_assert(far_smem_bytes<kMaxOrder, false>() <= 48 << 10, "dynamic shared memory without an opt-in");

template <int Q, bool LAB, bool MIXED, int FORM>
static void launch_far_q(const FarArgs &a, cudaStream_t s)
{
  far_kernel<Q, LAB, MIXED, FORM><<<far_blocks(a), 32 * kFarWarps, far_smem_bytes<Q, MIXED>(), s>>>(a);
}

template <int Q, bool LAB, bool MIXED, int FORM>
static void launch_far_batch_q(const FarArgs *args, const int *task_off, int n_ens, int blocks, cudaStream_t s)
{
  far_batch_kernel<Q, LAB, MIXED, FORM>
      <<<blocks, 32 * kFarWarps, far_smem_bytes<Q, MIXED>(), s>>>(args, task_off, n_ens);
}

// calls f<q>() for the run-time order
#define QG_BY_ORDER(q, CALL) \
  switch(q) {                \
    case 1: CALL(1); break;  \
    case 2: CALL(2); break;  \
    case 3: CALL(3); break;  \
    case 4: CALL(4); break;  \
    case 5: CALL(5); break;  \
    case 6: CALL(6); break;  \
    case 7: CALL(7); break;  \
    default: break;          \
  }

template <bool LAB, bool MIXED, int FORM>
static void launch_far_batch_frame(const FarArgs *args, const int *block_off, int n_ens, int blocks, int q,
                                   cudaStream_t s)
{
#define CALL(QQ) launch_far_batch_q<QQ, LAB, MIXED, FORM>(args, block_off, n_ens, blocks, s)
  QG_BY_ORDER(q, CALL)
#undef CALL
}

template <int FORM>
static void launch_far_batch_form(const FarArgs *args, const int *block_off, int n_ens, int blocks, int q, int frame,
                                  int mixed, cudaStream_t s)
{
  if(frame == 0)
    mixed ? launch_far_batch_frame<false, true, FORM>(args, block_off, n_ens, blocks, q, s)
          : launch_far_batch_frame<false, false, FORM>(args, block_off, n_ens, blocks, q, s);
  else
    mixed ? launch_far_batch_frame<true, true, FORM>(args, block_off, n_ens, blocks, q, s)
          : launch_far_batch_frame<true, false, FORM>(args, block_off, n_ens, blocks, q, s);
}

void launch_far_batch(const FarArgs *args, const int *block_off, const int *tile_off, int n_ens, int blocks, int tiles,
                      int q, int frame, int mixed, int form, void *stream)
{
  if(n_ens <= 0) return;
  cudaStream_t s = (cudaStream_t)stream;
  form == kFormPlain ? launch_far_batch_form<kFormPlain>(args, block_off, n_ens, blocks, q, frame, mixed, s)
                     : launch_far_batch_form<kFormAny>(args, block_off, n_ens, blocks, q, frame, mixed, s);
  far_reduce_batch_kernel<<<tiles, 32 * kTimeBlock, 0, s>>>(args, tile_off, n_ens);
}

template <bool LAB, bool MIXED>
static void launch_far_frame(const FarArgs &a, cudaStream_t s)
{
#define CALL(QQ)                                          \
  if(a.form == kFormPlain)                                \
    launch_far_q<QQ, LAB, MIXED, kFormPlain>(a, s);       \
  else                                                    \
    launch_far_q<QQ, LAB, MIXED, kFormAny>(a, s)
  QG_BY_ORDER(a.q, CALL)
#undef CALL
}

void launch_far(const FarArgs &a, void *stream)
{
  if(a.nT <= 0) return;
  cudaStream_t s = (cudaStream_t)stream;
  if(a.otf)
    launch_far_otf(a, stream);
  else if(a.frame == 0)
    a.mixed ? launch_far_frame<false, true>(a, s) : launch_far_frame<false, false>(a, s);
  else
    a.mixed ? launch_far_frame<true, true>(a, s) : launch_far_frame<true, false>(a, s);
  launch_far_reduce(a, kTimeBlock, stream);
}

// ---- one step ----------------------------------------------------------------------
// The far-pair field of one step (evaluations).  The table's stream from HBM
// bounds it, and each warp's entries are fetched AHEAD sources early in
// registers: what is in flight is that times the warps an SM holds, and a
// launch lasts whole waves of them (launch_far1_q chooses).  The same sums in
// the same order either way.
template <int Q, bool LAB, bool MIXED, int AHEAD>
__global__ void __launch_bounds__(32 * kFarWarps) far_step1_kernel(FarArgs a)
{
  const int lane = threadIdx.x & 31;
  const int task = blockIdx.x * kFarWarps + (threadIdx.x >> 5);
  const int t0 = *a.d_t0;
  if(blockIdx.x == 0 && threadIdx.x == 0) *a.far_t0_out = t0;
  if(task >= far_tasks(a)) return;  // uniform per warp
  const FarTask t = far_task(a, task);
  const int d_last = t0 + kWindow;
  const long long tile = (long long)t.I * a.nT;
  const int *dp = a.delay + tile * kTilePairs + lane;
  using C = std::conditional_t<MIXED, float2, typename FarAcc<LAB, 1>::C>;
  constexpr int N = MIXED ? Q + 2 : Q + 1;
  struct Pair {
    C c[N];
    int d;
  };
  auto load = [&](Pair &x, int s) {
    x.d = -1;
    if(s >= t.s1) return;
    x.d = __ldcs(dp + s * kTile);
    const long long e = (tile + s / kTile) * N * kTilePairs + (s % kTile) * kTile + lane;
#pragma unroll
    for(int i = 0; i < N; ++i) {
      if constexpr(MIXED)
        x.c[i] = __ldcs(a.coef32 + e + i * kTilePairs);
      else
        x.c[i] = FarAcc<LAB, 1>::load(a.coef + e + i * kTilePairs);
    }
  };
  std::conditional_t<MIXED, MixedAcc<LAB, Q, 1>, FarAcc<LAB, 1>> acc;
  acc.zero();
  auto take = [&](const Pair &x, int s) {
    if(x.d >= kTimeBlock && x.d <= d_last) {
      const int tau0 = t0 - x.d - Q, slot = wrap_slot(tau0, a.W);
      if constexpr(MIXED)
        window_conv_mixed<Q, LAB, 1, kFormAny>(a.ring32w + (long long)s * a.stride, a.ring32d + (long long)s * a.stride, slot,
                                     tau0, x.c, acc);
      else
        window_conv<Q, LAB, 1, kFormAny>(a.ring + (long long)s * a.stride, slot, tau0, x.c, acc);
    }
  };
  Pair x[AHEAD];
#pragma unroll
  for(int u = 0; u < AHEAD; ++u) load(x[u], t.s0 + u);
#pragma unroll 1
  for(int s = t.s0; s < t.s1; s += AHEAD) {
#pragma unroll
    for(int u = 0; u < AHEAD; ++u) {
      if constexpr(AHEAD == 2) {  // no third set of registers
        take(x[u], s + u);
        load(x[u], s + u + 2);
      } else {
        const Pair y = x[u];
        load(x[u], s + u + AHEAD);
        take(y, s + u);
      }
    }
  }
  store_partial<1>(a, t, acc);
}

// Blocks of the one-step kernel the device holds at once.
template <int Q, bool LAB, bool MIXED, int AHEAD>
static int far1_resident()
{
  static const int blocks = [] {
    int dev = 0, sms = 0, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, far_step1_kernel<Q, LAB, MIXED, AHEAD>, 32 * kFarWarps, 0);
    return std::max(1, sms * per);
  }();
  return blocks;
}

// Mixed: one source ahead, at every size (microseconds an evaluation at order
// 5, one against two ahead: 2048 dots 134 / 178, 4096 185 / 313, 5200 301 / 352).
// FP64: three ahead while all blocks then run at once (2048 dots 147 / 172,
// lab frame 143 / 178; past that 4096 dots 455 / 367), else two, or one where
// its smaller register count saves a wave (3500 dots 247 / 335, 5200 488 / 557;
// at equal waves, 4096 dots, 388 / 367).
template <int Q, bool LAB, bool MIXED>
static void launch_far1_q(const FarArgs &a, cudaStream_t s)
{
  const int blocks = far_blocks(a), threads = 32 * kFarWarps;
  if constexpr(MIXED) {
    far_step1_kernel<Q, LAB, true, 1><<<blocks, threads, 0, s>>>(a);
  } else {
    auto waves = [&](int resident) { return (blocks + resident - 1) / resident; };
    if(blocks <= far1_resident<Q, LAB, false, 3>())
      far_step1_kernel<Q, LAB, false, 3><<<blocks, threads, 0, s>>>(a);
    else if(waves(far1_resident<Q, LAB, false, 1>()) < waves(far1_resident<Q, LAB, false, 2>()))
      far_step1_kernel<Q, LAB, false, 1><<<blocks, threads, 0, s>>>(a);
    else
      far_step1_kernel<Q, LAB, false, 2><<<blocks, threads, 0, s>>>(a);
  }
}

template <bool LAB, bool MIXED>
static void launch_far1_frame(const FarArgs &a, cudaStream_t s)
{
#define CALL(QQ) launch_far1_q<QQ, LAB, MIXED>(a, s)
  QG_BY_ORDER(a.q, CALL)
#undef CALL
}

void launch_far_step1(const FarArgs &a, void *stream)
{
  if(a.nT <= 0) return;
  cudaStream_t s = (cudaStream_t)stream;
  if(a.otf)
    launch_far_otf_step1(a, stream);
  else if(a.frame == 0)
    a.mixed ? launch_far1_frame<false, true>(a, s) : launch_far1_frame<false, false>(a, s);
  else
    a.mixed ? launch_far1_frame<true, true>(a, s) : launch_far1_frame<true, false>(a, s);
  launch_far_reduce(a, 1, stream);
}

// ---- single-step evaluation without device allocation ----------------------
// Scratch of qg_history_evaluate_noalloc: one file-scope array, carved into
// the part partials, the reduced far field and two step indices.  Sized for
// at most kNoAllocMaxDots (padded) dots.
constexpr size_t kNoAllocPartialBytes = sizeof(double2) * kNoAllocMaxGroups * kNoAllocMaxDots;
constexpr size_t kNoAllocFieldBytes = sizeof(double2) * kNoAllocMaxDots;
constexpr size_t kNoAllocScratchBytes = kNoAllocPartialBytes + kNoAllocFieldBytes + 256;
static_assert(kNoAllocScratchBytes == kNoAllocScratchTotal, "scratch size");

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

// Device address of g_noalloc_scratch on the current device.  In host code the
// symbol is only a stand-in; the address comes from cudaGetSymbolAddress,
// looked up once per device (the first call on a device does it, so that
// call must precede any stream capture).
qg_status noalloc_scratch(NoAllocScratch *out)
{
  static std::mutex mu;
  static void *addr[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if(e != cudaSuccess) return qg_fail(QG_ERR_CUDA, "cudaGetDevice failed: %s", cudaGetErrorString(e));
  if(dev < 0 || dev >= 64) return qg_fail(QG_ERR_UNSUPPORTED, "device index %d beyond 63", dev);
  void *p = nullptr;
  {
    std::lock_guard<std::mutex> lock(mu);
    if(!addr[dev]) {
      e = cudaGetSymbolAddress(&addr[dev], g_noalloc_scratch);
      if(e != cudaSuccess) {
        addr[dev] = nullptr;
        return qg_fail(QG_ERR_CUDA, "cudaGetSymbolAddress(g_noalloc_scratch) failed: %s",
                       cudaGetErrorString(e));
      }
    }
    p = addr[dev];
  }
  unsigned char *b = (unsigned char *)p;
  out->partial = (double2 *)b;
  out->field = (double2 *)(b + kNoAllocPartialBytes);
  out->ints = (int *)(b + kNoAllocPartialBytes + kNoAllocFieldBytes);
  return QG_OK;
}

}  // namespace qg
