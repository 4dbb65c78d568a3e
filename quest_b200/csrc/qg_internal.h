// Internal declarations shared by the library's translation units.
#pragma once

#include <cmath>
#include <cstddef>
#include <cstdint>

#include <vector_types.h>  // double2

#include "../../include/quest_gpu.h"

// Records the message for qg_last_error() on this thread and returns code.
qg_status qg_fail(qg_status code, const char *fmt, ...);

namespace qg {

constexpr int kWindow = 22;      // History's negative-time extent (main.cpp:30)
constexpr int kCorrectorSteps = 10;  // NUM_CORRECTOR_STEPS (integrator.cpp:3)
constexpr int kMaxOrder = 7;     // largest interpolation order built
constexpr int kTimeBlock = 16;   // K: steps per pass of the far-pair kernel
constexpr int kRingMirror = 24;  // slots mirrored past the ring end (>= K+q)
constexpr int kTile = 32;        // dots per table tile (a warp's 32 targets)
constexpr int kTilePairs = kTile * kTile;
constexpr int kTileGroup = 4;    // source tiles per group of the far kernel
constexpr int kFarWarps = 4;     // warps (tasks) per far-kernel block
constexpr int kPcDepth = 23;     // PC ring: 22 past steps + the current one
constexpr int kBadNone = 0x7fffffff;

// Weights as passed to kernels (copy of qg_weights).
struct PCW {
  int n_time;
  double ps[64];
  double cs[64];
  double fc;
};

// Per-pair physics constants for coefficient kernels.
struct CoefParams {
  double c0, dt, mu0, hbar, omega;
  int q;
  int frame;
};

// The same constants as the on-the-fly kernels use them.
struct OtfConst {
  double c0dt, inv_c0dt;  // c0 dt and its correctly rounded reciprocal
  double c0, c0_sq, A;    // A = mu0 / (4 pi hbar)
  double inv_dt, inv_dt2;
  double om, om_sq;
  double half_turns, half_turns_low;  // omega / (pi c0) in two parts
};
inline OtfConst otf_const(const qg_params &p)
{
  OtfConst o;
  o.c0dt = p.c0 * p.dt;
  o.inv_c0dt = 1.0 / o.c0dt;
  o.c0 = p.c0;
  o.c0_sq = p.c0 * p.c0;
  o.A = p.mu0 / (4 * M_PI * p.hbar);
  o.inv_dt = 1.0 / p.dt;
  o.inv_dt2 = o.inv_dt * o.inv_dt;
  o.om = p.laser_frequency;
  o.om_sq = p.laser_frequency * p.laser_frequency;
  const long double ht = p.laser_frequency / (3.141592653589793238462643L * p.c0);
  o.half_turns = (double)ht;
  o.half_turns_low = (double)(ht - o.half_turns);
  return o;
}

struct PulseParams {
  double amp_pol[3];  // (amplitude / 2) * polarisation_k
  double k[3];        // wavevector
  double freq, delay, width;
};

// Arguments of the table-build kernel.
struct TableArgs {
  const double *pos;   // [n_pad][3] internal order
  const double *dip;   // [n_pad][3]
  const int *user;     // internal -> user index, -1 for padding
  int n, n_pad, nT;
  long long nblk;
  int *delay;          // [nT][nT][kTilePairs]
  double2 *coef;       // FP64: [nT][nT][q+1][kTilePairs]
  float2 *coef32;      // mixed: [nT][nT][q+2][kTilePairs] (taps, then their sum)
  int mixed;
  int *max_delay;      // atomicMax
  // [0] pairs with delay 0, [1] pairs with delay < K, [3] pairs with delay
  // >= K and a non-finite coefficient ([2] is the list builder's counter)
  unsigned long long *near_count;
  CoefParams cp;
};

// What a far launch knows of its windows.  kFormAny: nothing; samples before
// step -22 are skipped.  kFormPlain: no sample needs to be: every window starts
// at step -22 or later (blocks past the largest delay), or every coefficient
// is finite as it is held and the ring slots of steps before -22 still hold the
// zeros they were reset to (nothing but runs has written the history, and no
// captured call that would is about), whose products are +-0 and leave an accumulator that started at +0 bit for bit
// as it was.  Both forms give the same bits.  The plain form serves the first
// blocks too: testing or zeroing the dead samples there made a 640-step run
// of 4096 dots 2-4 % slower than it began, and the tests' registers cost the
// steady state as well (641 against 784 us a launch, zeroing).
enum : int { kFormAny = 0, kFormPlain = 1 };

// Arguments of the far-pair kernel: K steps of the pair sum for every pair
// with floor delay >= K, from one pass over the table (or one evaluation of
// the coefficients).
struct FarArgs {
  const int *delay;     // [nT][nT][kTilePairs] ordered tile pairs
  const double2 *coef;  // [nT][nT][q+1][kTilePairs]
  const double2 *ring;  // [n_pad][stride]: rho01 by time slot
  // mixed precision: FP32 table with the tap sum after the taps, and FP32
  // rings of rho01 and of its step-to-step differences (computed in FP64)
  const float2 *coef32;
  const float2 *ring32w;
  const float2 *ring32d;
  int mixed;
  double2 *partial;     // [K][nP][n_pad] per source part
  double2 *field;       // [K][n_pad] far-pair field
  int n_pad, nT, W, stride, q, frame;
  // sources: groups of `group` source tiles, each cut into `parts` parts of
  // `unit` sources (the last of a group may be shorter or empty); nP parts in
  // all.  A part's sum is one partial; the partials are added in part order.
  int group, parts, unit, nP;
  const int *d_t0;      // first step of the block
  int *far_t0_out;      // receives *d_t0 (read by the dot-step kernels)
  int form;             // what is known of the launch's windows: kFormAny or kFormPlain
  // on-the-fly coefficients (no table): dot data and constants
  int otf;
  const double *pos;    // [n_pad][3]
  const double *dip;    // [n_pad][3]
  const int *user;      // internal -> user index, -1 for padding
  OtfConst oc;
  // target tiles [tile_lo, tile_lo + tile_n) only (a shard of a sharded
  // handle; on-the-fly kernel); tile_n == 0: all nT
  int tile_lo, tile_n;
};

// Parts per source group (FarArgs::parts).  A far task, one warp's, is a
// target tile x one part, and 148 SMs hold 1776 at once (3 blocks of 4 warps).
// While there are fewer, a launch lasts one task, so the groups are cut until
// the tasks fill the device, or a part has 8 sources (beginning and ending a
// task cost about as much as 4).  The cut fixes the association of the far
// sums, so it depends on the ensemble and the group alone: the same alone, in
// a batch and in a shard.
inline int far_parts(int nT, int group)
{
  const long long tasks = (long long)nT * ((nT + group - 1) / group);
  const int n = group * kTile;
  int parts = 1;
  while(tasks * (parts + 1) <= 1776 && n / (parts + 1) >= 8) ++parts;
  return parts;
}

// A dot's state in the general step form (RowState, qg_step.cu), and the
// double2 per dot of StepArgs::scratch.
constexpr int kRowStateBytes = 160;
constexpr int kScratchPerDot = 2 + kRowStateBytes / 16;

// Arguments of the per-dot step kernels.
struct StepArgs {
  int n, n_pad, nT, W, stride, q, frame;
  int T;                 // num_timesteps: steps at or past T are not computed
  double dt, laser_freq, hbar;
  PulseParams pulse;
  const double *pos;     // [n_pad][3] internal order
  const double *dip;     // [n_pad][3]
  const double *freq, *t1, *t2;
  const int *user;       // internal -> user index, -1 for padding
  const double2 *far_field;  // [K][n_pad] far-pair field of the current block
  const int *far_t0;     // first step of the far block far_field holds
  // pairs with floor delay < K (taps not covered by the far kernel): CSR by
  // internal index, partner, delay and q+1 coefficients
  const int *mid_ptr;
  const int *mid_idx;
  const int *mid_delay;
  const double2 *mid_coef;  // [entry][q+1]
  // the mid-list taps that read step t-1 (delay 1 tap 0, delay 0 tap 1): CSR
  // by internal index, partner (internal index) and coefficient; lag = 1 when
  // every such partner is in the dot's own 32-dot block
  const int *new_ptr;
  const int *new_idx;
  const double2 *new_coef;
  int lag;
  int mid_cache;  // step-block kernel: mid-list entries a block keeps in shared memory
  // step-block kernel partner history: per 32-dot block its distinct mid-list
  // partners (CSR by block, internal indices), each entry's partner as an
  // index into its block's list, and the partners a block can hold (0: off)
  const int *bp_ptr;
  const int *bp_idx;
  const int *mid_pj;
  int hist_cap;
  // step-block kernel: per 32-dot block, the blocks holding its mid-list
  // partners, itself included (CSR by block)
  const int *pb_ptr;
  const int *pb_idx;
  double2 *pcr;          // [kPcDepth][4][n_pad]
  double2 *ring;         // [n_pad][stride] rho01 by step slot
  float2 *ring32w;       // mixed: FP32 rho01 by slot (null in FP64)
  float2 *ring32d;       // mixed: FP32 rho01(t) - rho01(t-1), differences in FP64
  // current-step coupling: CSR by slot (fused: partner = local slot in the
  // block; general: partner = internal index)
  const int *near_ptr;
  const int *near_idx;
  const double2 *near_coef;
    double2 *scratch;      // general form: [2][n_pad] iterates exchanged by its grid, then kRowStateBytes a dot
  double2 *traj;         // [k][n][2] user order or null
  int traj_rows;         // rows allocated in traj
  const int *traj_t0;    // the step of row 0 (null: traj_base)
  int traj_base;
  int *d_next;           // first step of the next far block (set by the last
                         // step kernel of a block, read by the far kernel)
  int *d_bad;
  // step-block kernel and the general form's grid: polls per wait on other
  // blocks before it gives up (0: the default, about a second), and a block
  // that never posts (-1: none; set only by failure-detection tests, so that
  // waits run out)
  int spin_limit;
  int skip_post_block;
  int blk_lo;  // first 32-dot block of the per-step launch (a shard's range)
  PCW w;
};

// A dot's run of the mid list: its entries' partners and delays, its
// coefficients (q + 1 per entry) and how many of those there are.  Offsets into
// the lists are ints, but an offset times q + 1 need not fit one: a group of
// 16 400 dots coupled to one another has 2^28 entries, whose coefficients at
// q = 7 are 2^31.
struct MidRow {
  const int *idx, *delay;
  const double2 *coef;
  int taps;
};
__host__ __device__ inline MidRow mid_row(const StepArgs &a, int dot)
{
  const int e0 = a.mid_ptr[dot], e1 = a.mid_ptr[dot + 1], q1 = a.q + 1;
  return MidRow{a.mid_idx + e0, a.mid_delay + e0, a.mid_coef + (long long)e0 * q1, (e1 - e0) * q1};
}

// Whether the lists of `pairs` pairs with floor delay < K, an entry for each
// dot of a pair, can be addressed: their offsets are ints.
inline bool mid_list_fits(unsigned long long pairs) { return pairs <= 0x7fffffffULL / 2; }

// Scratch of the allocation-free evaluation (qg_history_evaluate_noalloc):
// a static device array in qg_far.cu, at most kNoAllocMaxDots padded dots.
// Uncut, the partials are kNoAllocMaxGroups x n_pad at most; where far_parts
// cuts the groups there are 1776 tasks at most, 1776 x 32 values.
constexpr int kNoAllocMaxDots = 4096;
constexpr int kNoAllocMaxTiles = kNoAllocMaxDots / kTile;
constexpr int kNoAllocMaxGroups = (kNoAllocMaxTiles + kTileGroup - 1) / kTileGroup;
constexpr size_t kNoAllocScratchTotal = 16ull * kNoAllocMaxGroups * kNoAllocMaxDots + 16ull * kNoAllocMaxDots +
                                        256;
struct NoAllocScratch {
  double2 *partial;    // [nP][n_pad], room for kNoAllocMaxGroups * kNoAllocMaxDots
  double2 *field;      // [n_pad]
  int *ints;           // [0] step, [1] far_t0 written by the kernel
};
qg_status noalloc_scratch(NoAllocScratch *out);
// The far field of one step (slice 0 of the field): evaluations
void launch_far_step1(const FarArgs &a, void *stream);
// Many ensembles: block_off[e] = first far block of ensemble e (far_blocks of
// each), tile_off[e] = its first 32-dot tile; totals at [n_ens]
void launch_far_batch(const FarArgs *args, const int *block_off, const int *tile_off, int n_ens, int blocks, int tiles,
                      int q, int frame, int mixed, int form, void *stream);
void launch_ring32_rebuild(const StepArgs &a, void *stream);
// *out = 1 if any ring (FP64, and FP32 in mixed precision) holds a non-zero in slots [lo, hi)
void launch_ring_nonzero(const StepArgs &a, int lo, int hi, int *out, void *stream);
// Sharded handles: a shard's rho01 at step t for internal dots [lo, hi)
// into out[0 .. hi-lo), and the other dots' rho01 at step t from the full
// internal-order vector into the rings (as the step kernel writes its own)
void launch_shard_export(const StepArgs &a, int t, int lo, int hi, double2 *out, void *stream);
void launch_shard_import(const StepArgs &a, int t, int lo, int hi, const double2 *full, void *stream);
// out[e] = *args[e].d_bad for the n members of a batch
void launch_gather_bad(const StepArgs *args, int n, int *out, void *stream);
// The step-block kernel's per-block step counts, one per 128-byte line (so
// the polls on one block's count do not queue behind those on another's).
constexpr int kFlagStride = 32;
void launch_step_block(const StepArgs &a, int k0, int k1, int nblocks, unsigned *flags, void *stream);
// The general step form's launch: one cluster or a cooperative grid of
// `blocks` blocks of `rows` dots, `cache` near entries in shared memory,
// stage: the iterates copied there, state: the rows' states kept there
struct GroupShape {
  int cluster, blocks, rows, cache, stage, state;
  size_t smem;
};
GroupShape group_shape(int n_pad, const int *near_ptr);
void launch_step_group(const StepArgs &a, int k0, int k1, const GroupShape &g, unsigned *counter, void *stream);
int step_block_max_blocks(int q, int mid_cache, int hist_cap);
// pipe: the mid list staged with several entries' loads in flight (same sums)
void launch_step_batch(const StepArgs *args, const int *block_off, int n_ens, int total_blocks, int n_time,
                       int k, bool pipe, void *stream);

// Far-kernel tasks (warps) of one ensemble, and the blocks that hold them.
__host__ __device__ inline int far_tasks(const FarArgs &a) { return (a.tile_n > 0 ? a.tile_n : a.nT) * a.nP; }
inline int far_blocks(const FarArgs &a) { return (far_tasks(a) + kFarWarps - 1) / kFarWarps; }

// Launchers (defined in the .cu files).
void launch_table_build(const TableArgs &a, int q, void *stream);
void launch_far(const FarArgs &a, void *stream);
void launch_far_otf(const FarArgs &a, void *stream);
void launch_far_otf_step1(const FarArgs &a, void *stream);
// field[k][.] = the sum of the partials over the parts, in part order, for k < steps
void launch_far_reduce(const FarArgs &a, int steps, void *stream);
// whole: += far pairs at a whole delay (fraction 0)
void launch_max_delay(const double *pos, const int *user, int n_pad, double c0dt, int *max_delay,
                      unsigned long long *whole, void *stream);
void launch_near_find(const double *pos, const int *user, int n_pad, double c0dt, int below, int *out_pairs,
                      unsigned long long *counter, unsigned long long cap, void *stream);
void launch_pair_list_coef(const TableArgs &a, int q, const int *pairs, long long m, double2 *out, void *stream);
// dst[j][0 .. width) = src[rows[j]][0 .. width), j < n
void launch_gather_rows(const double2 *src, const long long *rows, int width, long long n, double2 *dst,
                        void *stream);
void launch_step_fused(const StepArgs &a, int k, int nblocks, void *stream);
void launch_eval_field(const StepArgs &a, const int *d_eval_step, double2 *out_user, void *stream);
void launch_pulse_field(const StepArgs &a, int step, double2 *out_user, void *stream);
void launch_set_int(int *p, int v, void *stream);
void launch_init_state(const StepArgs &a, void *stream);
void launch_ring_write(const StepArgs &a, int t, const double2 *rho01_user, void *stream);
void launch_ring_read(const StepArgs &a, int t, double2 *rho01_user, void *stream);
void launch_state_read(const StepArgs &a, int t, double2 *rho_user, void *stream);

}  // namespace qg
