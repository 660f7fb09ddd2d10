// Device code that decides how a batch is cut: the scan of the prepare blocks' counts with the choice
// of window mode (k_prep_scan), the window list of a layered job (cut_windows), the planner of the
// fused kernel's work items (k_plan, k_plan_write) and when a CTA empties its table (cta_over).
// Integer arithmetic, warp and CTA steps only, no inline assembly: the CPU tests compile this header
// with the host compiler and run it under other orders of the warps than a GPU happens to take.
#pragma once
#include <limits.h>
#include "st_device.cuh"

namespace st {

// Start of a kernel that may be launched by launch_chained: the next kernel of the chain may be put
// on the SMs from here on, and this one waits for the end of the one before it (and so of all
// before that: each of them waited likewise) before it reads or writes anything.
__device__ __forceinline__ void chain_start() {
  cudaTriggerProgrammaticLaunchCompletion();
  cudaGridDependencySynchronize();
}

// A windowed job whose kept deposits share cells (fewer than half as many occupied flag cells
// of side d as deposits, or a quarter as many of side 2d: several hits per sphere) runs with
// coarse windows of kCoarseTiles warp tiles per warp; others with kWinTiles. Its cells record
// windows of kWindow deposits, a coarse window is two of them.
__device__ __forceinline__ bool coarse_windows(const JobDev& J, const JobAux& A) {
  return A.windowed == kWinFlags && (J.cell_nbr8 ? 4 : 2) * (long long)A.cells < A.kept;
}

// A bin belongs to one CTA per oversample, so in a launch with too few oversamples to go round, a
// layered job takes as long as its largest bin, while boundary flags spread an oversample over the
// CTAs by chunks. Measured there (one track, 148 CTAs): layers 0.1 ms + 0.95 ns per deposit of the
// largest bin, flags 0.6 ns per kept deposit. Dense tracks across z, layers / flags, fused: 1e6
// deposits, 30 nm, 4 oversamples (nearly all in one bin) 0.80 / 0.48 ms; 300,007, 30 nm, 10 (two
// bins) 0.27 / 0.15; 600,000, 20 nm, 10 (two) 0.31 / 0.34; 2e6, 20 nm, 4 (two) 0.90 / 1.25; 4e6,
// 10 nm, 4 (two) 1.99 / 2.56. With CTAs enough at work, layers take three quarters of flags' time.
// (Chunks of a layered bin that meet in a spill table took 4.2 ms on the last one.)
__device__ __forceinline__ bool one_bin_too_large(const PrepareParams& p, long long kept,
                                                  long long largest) {
  const long long fixed = 84 << 10;
  return kept > p.unit_min && 3 * largest > kept && 100 * (largest + fixed) > 63 * kept &&
         10 * (largest + fixed) > 13 * p.cta_share;
}

// One CTA per job: exclusive scan of the job's block counts.
__global__ void __launch_bounds__(1024) k_prep_scan(PrepareParams p) {
  chain_start();
  const int j = blockIdx.x;
  const int64_t b0 = p.blk_prefix[j], nb = p.blk_prefix[j + 1] - b0;
  __shared__ long long s_warp[32];
  __shared__ long long s_carry;
  if (threadIdx.x == 0) s_carry = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int64_t base = 0; base < nb; base += 1024) {
    const int64_t k = base + threadIdx.x;
    long long v = k < nb ? p.blk_count[b0 + k] : 0;
    long long incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      long long w = s_warp[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const long long t = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += t;
      }
      s_warp[lane] = w;  // inclusive over warps
    }
    __syncthreads();
    const long long warp_base = warp ? s_warp[warp - 1] : 0;
    if (k < nb) p.blk_offset[b0 + k] = s_carry + warp_base + incl - v;
    __syncthreads();
    if (threadIdx.x == 0) s_carry += s_warp[31];
    __syncthreads();
  }
  const long long kept = s_carry;
  const bool many = kept > p.flag_min_kept && !(p.aux[j].flags & kAuxWraps);
  int mode = p.jobs[j].flagged && many ? kWinFlags : kWinNone;
  if (p.jobs[j].layers && many) {
    // the bin counts to first places, and the deposits that lie in bins larger than a window
    uint32_t* bins = p.bins + p.jobs[j].bin_off;
    const int nb = p.jobs[j].n_bins;
    constexpr int kPer = kMaxBins / 1024;
    unsigned v[kPer], sum = 0, big = 0, most = 0;
#pragma unroll
    for (int t = 0; t < kPer; ++t) {
      const int b = (int)threadIdx.x * kPer + t;
      v[t] = b < nb ? bins[b] : 0;
      sum += v[t];
      big += v[t] > (unsigned)(2 * kWindow) ? v[t] : 0;
      most = max(most, v[t]);
    }
    unsigned incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    __shared__ unsigned s_bin[32];
    __shared__ unsigned long long s_big;
    __shared__ unsigned s_most;
    if (threadIdx.x == 0) {
      s_big = 0;
      s_most = 0;
    }
    if (lane == 31) s_bin[warp] = incl;
    __syncthreads();
    if (big) atomicAdd(&s_big, (unsigned long long)big);
    if (most) atomicMax(&s_most, most);
    unsigned base = incl - sum;
    for (int w = 0; w < warp; ++w) base += s_bin[w];
#pragma unroll
    for (int t = 0; t < kPer; ++t) {
      const int b = (int)threadIdx.x * kPer + t;
      if (b < nb) bins[b] = base;
      base += v[t];
    }
    __syncthreads();
    // Layers unless more than a quarter of the deposits lie in bins of over two windows (a track
    // across z): such bins empty into the spill log piece by piece, where windows along the track
    // would leave few boundary spheres. On dense tracks (over 1,024 deposits per sphere diameter
    // of track length) a window along the track is hardly longer than a sphere, and the spheres
    // of a large bin fit the table. Fused time of 8 ion tracks, layers / flags: along z, 1e6
    // deposits, 2 nm 7.3 / 12.1 ms; across z, 1e6, 2 nm (sparse) 13.2 / 9.6, 1e6, 10 nm (1,000
    // per diameter) 5.5 / 5.4, 4e6, 10 nm (4,000) 9.4 / 13.5, 2e6, 20 nm (8,000) 3.5 / 7.6.
    const JobDev& J = p.jobs[j];
    const bool dense = (double)J.n * J.d > 1024.0 * 2.0 * J.HL;
    const bool layers = dense || 4 * s_big <= (unsigned long long)kept;
    if (mode == kWinNone || (layers && !one_bin_too_large(p, kept, s_most))) mode = kWinLayers;
  }
  if (threadIdx.x == 0) {
    p.aux[j].kept = kept;
    p.aux[j].windowed = mode;
    if (mode == kWinFlags) *p.any_flags = 1;
  }
}

// Window list of a layered job, by one warp: from the first place k0 of a window, whose tile span
// ends at `limit`, the window ends after one of the bins that end by then, or at `limit` when the
// bin itself goes on (its next window is marked kWinContinues). bins[b] is the end of bin b.
//
// Size: a window of win_tiles holds as many cells as the table has slots when every deposit has a
// cell of its own, and fills about 30 % of it with spheres. Denser jobs (m deposits per cell, counted
// per prepare block) get m times the tiles, up to eight times: fewer barriers, and more rounds over
// which the warps' work evens out. From four times on the end is the bin that wastes least of the
// last round of one tile per warp, a window costing about three quarters of a round besides; short
// windows take all the bins that fit. Large bins left windows of 39 tiles for 32 warps, which
// waited for 38 % of the time: 8 tracks of 4e6 deposits, 10 nm, fused 20.8 -> 18.1 ms with the
// binning below (21.8 -> 18.7 without it).
__device__ __forceinline__ void cut_windows(const PrepareParams& p, const JobDev& J, JobAux* aux,
                                            const uint32_t* bins) {
  const int lane = threadIdx.x;
  unsigned long long* wins = p.wins + J.win_off;
  const long long kept = aux->kept;
  const long long cells = (long long)aux->cells > 0 ? (long long)aux->cells : 1;
  const long long m = kept / cells;
  const long long tiles = (m < 2 ? 1 : m < 4 ? 2 : m > 8 ? 8 : m) * p.win_tiles;
  long long k0 = 0;
  unsigned long long mark = 0;
  int n = 0, b = 0;  // b: first bin that ends behind k0
  while (k0 < kept) {
    if (lane == 0) wins[n] = (unsigned long long)k0 | mark;
    ++n;
    const long long limit = (k0 / kWarpTile + tiles) * kWarpTile;
    long long end = k0;
    unsigned best = 0;
    for (int c = b;; c += 32) {
      const long long e = c + lane < J.n_bins ? (long long)bins[c + lane] : LLONG_MAX;
      const unsigned in = __ballot_sync(0xffffffffu, e <= limit);  // a prefix of the lanes
      unsigned score = 0;
      if (e <= limit && e > k0) {
        const unsigned t = (unsigned)((e + kWarpTile - 1) / kWarpTile - k0 / kWarpTile);
        const unsigned rounds = (t + kFusedWarps - 1) / kFusedWarps;
        score = m < 4 ? t : (t * 4096 / (4 * rounds + 3)) << 12 | (t & 0xFFF);
      }
      const unsigned top = __reduce_max_sync(0xffffffffu, score);
      if (top && top >= best) {  // (equal: further bins inside the same tile)
        const int w = 31 - __clz(__ballot_sync(0xffffffffu, score == top));
        best = top;
        end = __shfl_sync(0xffffffffu, e, w);
        b = c + w + 1;
      }
      if (in != 0xffffffffu) break;
    }
    if (end > k0) {
      k0 = end;
      mark = 0;
    } else {
      k0 = limit;
      mark = kWinContinues;
    }
  }
  if (lane == 0) {
    wins[n] = (unsigned long long)kept;
    aux->n_win = n;
  }
}

// A barrier of the CTA that returns, in every thread, whether a shared count that threads add to on
// their way to it ends above `limit`. Whoever adds last sees the final count before arriving; a read
// after a plain barrier would race with the additions of threads that are already past it, and
// threads could part ways there.
__device__ __forceinline__ bool cta_over(const int* count, int limit) {
  return __syncthreads_or(*(const volatile int*)count > limit) != 0;
}

// ---------------------------------------------------------------------------------------------
// Planner (after the prepare stage, before k_fused): work items from the kept deposit counts.
// A job whose kept deposits per oversample exceed both min_chunks chunks (4) and 1/share_divisor
// (1/8) of one CTA's share of the batch runs as shared units (one per oversample, `helpers` helper items each);
// every other job runs as private items (plan_item_cost), a layered job's also as parts of an
// oversample. Items are
// bucketed by cost, largest first (longest-processing-time order at bucket granularity).
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ int cost_bucket(long long cost) {
  int l = 0;
  while (cost > 1 && l < 62) { cost >>= 1; ++l; }
  return kPlanBuckets - 1 - l;  // larger cost -> smaller bucket -> earlier
}

// Work of one item: item_cost, or an eighth of a CTA's share of a batch too small for that, down
// to 2,048 deposit*oversamples (half of a warp tile per warp; smaller items cost as much). With
// items of item_cost a single proton track of 100 oversamples ran on 3 of the 148 CTAs: fused
// 0.40 ms, against 0.062 ms split; a track of 10 oversamples, one at a time, 84 -> 25 us. A half
// instead of an eighth of the share made groups of uneven tracks wait for their largest items
// (6.2 against 5.6 ms for 256 host tracks in groups).
__device__ __forceinline__ long long plan_item_cost(const PlanParams& q, unsigned long long total_units) {
  const long long share = (long long)(total_units / ((unsigned long long)q.grid * 8));
  const long long lo = 2048;
  const long long ic = share < lo ? lo : share;
  return ic < q.item_cost ? ic : q.item_cost;
}

__device__ __forceinline__ JobPlan plan_job(const PlanParams& q, int j, unsigned long long total_units) {
  const long long kept = q.aux[j].kept;
  const long long nos = q.jobs[j].n_os;
  JobPlan pl;
  pl.items = 0;
  pl.bucket = kPlanBuckets - 1;
  pl.unit_base = -1;
  pl.blk_os = 1;
  pl.blk_win = 0;
  if (kept > 0 && nos > 0 && !(q.aux[j].flags & kAuxNonfinite)) {
    const long long chunk = chunk_tiles(q.chunk_windows) * kWarpTile;
    const long long share =
        q.share_divisor > 0 ? (long long)(total_units / ((unsigned long long)q.share_divisor * q.grid)) : 0;
    if (q.aux[j].windowed == kWinLayers) {
      // any range of windows is complete on its own: about item_cost of work per item, as whole
      // oversamples or as parts of one
      const long long n_win = q.aux[j].n_win;
      const long long ic = plan_item_cost(q, total_units);
      if (kept > ic && n_win > 1) {
        long long parts = (kept + ic - 1) / ic;
        parts = parts < q.max_helpers ? parts : q.max_helpers;
        parts = parts < n_win ? parts : n_win;
        const long long per = (n_win + parts - 1) / parts;
        pl.blk_win = (int)per;
        pl.blk_os = 1;
        pl.items = (int)(nos * ((n_win + per - 1) / per));
        pl.bucket = cost_bucket(kept / parts);
      } else {
        long long b = ic / kept;
        b = b < 1 ? 1 : (b > nos ? nos : b);
        pl.blk_os = (int)b;
        pl.items = (int)((nos + b - 1) / b);
        pl.bucket = cost_bucket(kept * b);
      }
    } else if (q.share_divisor > 0 && kept > (long long)q.min_chunks * chunk && kept > share) {
      const long long chunks = (kept + chunk - 1) / chunk;
      const int helpers = (int)(chunks < q.max_helpers ? chunks : q.max_helpers);
      pl.blk_os = helpers;
      pl.items = (int)(nos * helpers);
      pl.unit_base = (int)atomicAdd(q.unit_counter, (unsigned)nos);
      pl.bucket = cost_bucket(kept);
    } else {
      const long long pad = ((kept + kWarpTile - 1) / kWarpTile) * kWarpTile;
      long long b = plan_item_cost(q, total_units) / pad;
      b = b < 1 ? 1 : (b > nos ? nos : b);
      pl.blk_os = (int)b;
      pl.items = (int)((nos + b - 1) / b);
      pl.bucket = cost_bucket(pad * b);
    }
  }
  return pl;
}

// Items of job j, by the threads i = first, first + step, ... of the caller, from position `at`.
__device__ __forceinline__ void plan_items(const PlanParams& q, int j, const JobPlan& pl, long long at,
                                           int first, int step) {
  const int nos = q.jobs[j].n_os;
  for (int k = first; k < pl.items; k += step) {
    const long long pos = at + k;
    if (pos >= q.item_cap) break;
    WorkItem w;
    w.job = j;
    if (pl.blk_win > 0) {
      const int parts = (q.aux[j].n_win + pl.blk_win - 1) / pl.blk_win;
      w.os_begin = k / parts;
      w.os_count = -pl.blk_win;
      w.unit = -1 - k % parts;
    } else if (pl.unit_base >= 0) {
      const int u = k / pl.blk_os;
      w.os_begin = u;
      w.os_count = 1;
      w.unit = pl.unit_base + u;
    } else {
      w.os_begin = k * pl.blk_os;
      w.os_count = (w.os_begin + pl.blk_os <= nos) ? pl.blk_os : nos - w.os_begin;
      w.unit = -1;
    }
    q.items[pos] = w;
  }
}

// One CTA: the batch's work, every job's plan, the buckets' places in the item list and, for up to
// kPlanSmall jobs, the items themselves (k_plan_write writes those of larger batches). One launch
// instead of the four that these steps were: a dependent launch costs a small batch 3 to 5 us.
// With k_reset for the memsets: one proton track of 19,997 deposits 214 -> 181 us per pass, 16 short
// tracks one at a time 2.10 -> 1.63 ms, 64 in a batch 286 -> 269 us.
constexpr int kPlanSmall = 64;
__global__ void __launch_bounds__(1024) k_plan(PlanParams q) {
  chain_start();
  __shared__ unsigned long long s_total;
  // (cursors of their own: warp 0 still reads the counts when the other warps are past the scan)
  __shared__ unsigned s_count[kPlanBuckets], s_start[kPlanBuckets], s_cursor[kPlanBuckets];
  const int tid = threadIdx.x, lane = tid & 31;
  if (tid == 0) s_total = 0;
  if (tid < kPlanBuckets) s_count[tid] = s_cursor[tid] = 0;
  __syncthreads();
  unsigned long long v = 0;
  for (int j = tid; j < q.n_jobs; j += 1024)
    v += (unsigned long long)q.aux[j].kept * (unsigned long long)q.jobs[j].n_os;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (lane == 0 && v) atomicAdd(&s_total, v);
  __syncthreads();
  const unsigned long long total = s_total;
  for (int j = tid; j < q.n_jobs; j += 1024) {
    const JobPlan pl = plan_job(q, j, total);
    q.plan[j] = pl;
    if (pl.items) atomicAdd(&s_count[pl.bucket], (unsigned)pl.items);
  }
  __syncthreads();
  if (tid < 32) {  // exclusive scan of the buckets, two per lane
    static_assert(kPlanBuckets == 64, "two buckets per lane");
    const unsigned a = s_count[2 * lane], b = s_count[2 * lane + 1];
    unsigned incl = a + b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    const unsigned base = incl - a - b;
    s_start[2 * lane] = base;
    s_start[2 * lane + 1] = base + a;
    q.bucket_start[2 * lane] = base;
    q.bucket_start[2 * lane + 1] = base + a;
    if (lane == 31) *q.n_items = (long long)incl <= q.item_cap ? (int)incl : (int)q.item_cap;
  }
  if (q.n_jobs > kPlanSmall) return;
  __syncthreads();
  for (int j = tid >> 5; j < q.n_jobs; j += 32) {
    const JobPlan pl = q.plan[j];
    if (pl.items == 0) continue;
    unsigned at = 0;
    if (lane == 0) at = s_start[pl.bucket] + atomicAdd(&s_cursor[pl.bucket], (unsigned)pl.items);
    at = __shfl_sync(0xffffffffu, at, 0);
    plan_items(q, j, pl, at, lane, 32);
  }
}

__global__ void __launch_bounds__(128) k_plan_write(PlanParams q) {
  chain_start();
  const int j = blockIdx.x;
  const JobPlan pl = q.plan[j];
  if (pl.items == 0) return;
  __shared__ unsigned s_pos;
  if (threadIdx.x == 0)
    s_pos = q.bucket_start[pl.bucket] + atomicAdd(&q.bucket_cursor[pl.bucket], (unsigned)pl.items);
  __syncthreads();
  plan_items(q, j, pl, s_pos, threadIdx.x, 128);
}

}  // namespace st
