// The kernels of planning.cuh on the host (cta_emulator.h) and host functions of st_device.cuh, as a
// library for test_planning_on_cpu.py.
#include "cta_emulator.h"
// (after the emulator's intrinsics)
#include "../supertrack_b200/csrc/planning.cuh"

#include <cmath>
#include <cstring>

namespace {
std::vector<int> warps(int n, const int32_t* order) { return std::vector<int>(order, order + n); }
}  // namespace

extern "C" {

// Plans a batch of jobs (kept deposits, oversamples and, for layered jobs, windows of each) as the
// library does; items_out: {job, os_begin, os_count, unit} per entry. Returns the number of items
// that k_plan publishes.
int plan_batch(int n_jobs, const int64_t* kept, const int32_t* n_os, const int32_t* n_win, int grid, int64_t item_cost,
               int share_divisor, int64_t item_cap, const int32_t* order, int32_t* items_out) {
  std::vector<st::JobDev> jobs(n_jobs);
  std::vector<st::JobAux> aux(n_jobs);
  std::vector<st::JobPlan> plan(n_jobs);
  std::vector<st::WorkItem> items(item_cap);
  std::memset(items.data(), 0xFF, items.size() * sizeof(st::WorkItem));
  for (int j = 0; j < n_jobs; ++j) {
    std::memset(&jobs[j], 0, sizeof(st::JobDev));
    std::memset(&aux[j], 0, sizeof(st::JobAux));
    jobs[j].n = kept[j];
    jobs[j].n_os = n_os[j];
    aux[j].kept = kept[j];
    aux[j].n_win = n_win[j];
    aux[j].windowed = n_win[j] > 0 ? st::kWinLayers : st::kWinNone;
  }
  unsigned start[st::kPlanBuckets] = {}, cursor[st::kPlanBuckets] = {}, unit = 0;
  int n_items = 0;
  st::PlanParams q;
  std::memset(&q, 0, sizeof(q));
  q.jobs = jobs.data();
  q.aux = aux.data();
  q.n_jobs = n_jobs;
  q.chunk_windows = 4;
  q.max_helpers = 32;
  q.grid = grid;
  q.item_cost = item_cost;
  q.share_divisor = share_divisor;
  q.min_chunks = 4;
  q.bucket_start = start;
  q.bucket_cursor = cursor;
  q.unit_counter = &unit;
  q.plan = plan.data();
  q.items = items.data();
  q.n_items = &n_items;
  q.item_cap = item_cap;
  emu::run_cta(1024, dim3(1), 0, warps(32, order), [&] { st::k_plan(q); });
  if (n_jobs > st::kPlanSmall)
    for (int j = 0; j < n_jobs; ++j)
      emu::run_cta(128, dim3(n_jobs), j, warps(4, order + 32), [&] { st::k_plan_write(q); });
  for (int64_t i = 0; i < item_cap; ++i) {
    const st::WorkItem& w = items[i];
    const int32_t v[4] = {w.job, w.os_begin, w.os_count, w.unit};
    std::memcpy(items_out + 4 * i, v, sizeof(v));
  }
  return n_items;
}

// Window mode that k_prep_scan gives a job with these z bins (the kept deposits of all); the bins
// become their first places.
int window_mode(int n_bins, uint32_t* bins, double per_diameter, int64_t cta_share, int64_t unit_min,
                const int32_t* order) {
  st::JobDev job;
  st::JobAux aux;
  st::PrepareParams p;
  std::memset(&job, 0, sizeof(job));
  std::memset(&aux, 0, sizeof(aux));
  std::memset(&p, 0, sizeof(p));
  int64_t kept = 0;
  for (int b = 0; b < n_bins; ++b) kept += bins[b];
  const int blocks = (int)((kept + 1023) / 1024);
  std::vector<int32_t> count(blocks, 1024);
  if (blocks) count.back() = (int32_t)(kept - (blocks - 1) * 1024ll);
  std::vector<int64_t> offset(blocks);
  const int64_t prefix[2] = {0, blocks};
  int32_t any = 0;
  job.n = kept;
  job.d = per_diameter / kept;  // n * d / (2 HL) deposits per sphere diameter
  job.HL = 0.5;
  job.flagged = job.layers = 1;
  job.n_bins = n_bins;
  p.jobs = &job;
  p.aux = &aux;
  p.n_jobs = 1;
  p.blk_prefix = prefix;
  p.blk_count = count.data();
  p.blk_offset = offset.data();
  p.bins = bins;
  p.any_flags = &any;
  p.flag_min_kept = 16384;
  p.cta_share = cta_share;
  p.unit_min = unit_min;
  emu::run_cta(1024, dim3(1), 0, warps(32, order), [&] { st::k_prep_scan(p); });
  for (int b = 0; b < blocks; ++b)
    if (offset[b] != b * 1024ll) return -1;
  return aux.kept == kept && any == (aux.windowed == st::kWinFlags) ? aux.windowed : -2;
}

// The window list that cut_windows makes of a job's z bins (their ends) with `cells` occupied cells:
// n_win + 1 entries. Returns n_win.
int cut(int n_bins, const uint32_t* ends, int64_t cells, int win_tiles, uint64_t* wins) {
  st::JobDev job;
  st::JobAux aux;
  st::PrepareParams p;
  std::memset(&job, 0, sizeof(job));
  std::memset(&aux, 0, sizeof(aux));
  std::memset(&p, 0, sizeof(p));
  job.n_bins = n_bins;
  aux.kept = ends[n_bins - 1];
  aux.cells = cells;
  p.win_tiles = win_tiles;
  static_assert(sizeof(unsigned long long) == sizeof(uint64_t), "");
  p.wins = reinterpret_cast<unsigned long long*>(wins);
  emu::run_cta(32, dim3(1), 0, {0}, [&] { st::cut_windows(p, job, &aux, ends); });
  return aux.n_win;
}

// The integer geometry of deposits (x, y) and their z offsets dz in an oversample of shift (sx, sy),
// with the constants of set_integer_geometry and the float steps of the fused kernel: bit 0 in the
// voxel, bit 1 a hit, bit 2 left to FP64, and the sphere's indices. Returns g_shift.
int integer_geometry(int n, int64_t lattice, double d, double gso, double sx, double sy, const double* x,
                     const double* y, const double* dz, int32_t* decision, int32_t* kx, int32_t* ky) {
  st::JobDev J;
  std::memset(&J, 0, sizeof(J));
  J.N = (uint32_t)lattice;
  J.d = d;
  st::set_integer_geometry(&J);
  const int half = 1 << J.g_shift >> 1;
  const int cx = (int)std::nearbyint((sx - gso) * J.g_scale) + half;
  const int cy = (int)std::nearbyint((sy - gso) * J.g_scale) + half;
  const unsigned in_max = (unsigned)J.g_ns - 4u, near_max = (unsigned)J.g_ns + 2u, low = (1u << J.g_shift) - 1u;
  const float centre = 8388608.0f + (float)(1 << J.g_shift) * 0.5f;
  const auto offset = [&](unsigned v) {
    const unsigned bits = (v & low) | 0x4B000000u;
    float f;
    std::memcpy(&f, &bits, 4);
    return f - centre;
  };
  for (int i = 0; i < n; ++i) {
    const unsigned vx = (unsigned)(int)std::nearbyint(x[i] * J.g_scale) + (unsigned)cx;
    const unsigned vy = (unsigned)(int)std::nearbyint(y[i] * J.g_scale) + (unsigned)cy;
    const double gz = dz[i] * J.g_scale;
    const float z2 = (float)(gz * gz);
    const bool in = vx - 2u <= in_max && vy - 2u <= in_max;
    const bool near = vx + 1u <= near_max && vy + 1u <= near_max;
    const float fx = offset(vx), fy = offset(vy);
    const float d2 = std::fma(fx, fx, std::fma(fy, fy, z2));
    const bool hit = in && d2 <= J.g_lo;
    const bool open = in ? (!hit && d2 <= J.g_hi) : near;
    decision[i] = (in ? 1 : 0) | (hit ? 2 : 0) | (open ? 4 : 0);
    kx[i] = (int)vx >> J.g_shift;
    ky[i] = (int)vy >> J.g_shift;
  }
  return J.g_shift;
}

// Windows of a CTA that adds `per_window` to a count in each and empties it above `limit` (cta_over).
// Returns how many threads took another branch than thread 0 at some window's end.
int empty_windows(int windows, int per_window, int limit, const int32_t* order) {
  static int count;
  static unsigned long long took[1024];
  count = 0;
  emu::run_cta(1024, dim3(1), 0, warps(32, order), [&] {
    const int tid = threadIdx.x;
    took[tid] = 0;
    for (int w = 0; w < windows; ++w) {
      if (tid < per_window) atomicAdd(&count, 1);
      if (st::cta_over(&count, limit)) {
        took[tid] |= 1ull << w;
        __syncthreads();
        if (tid == 0) count = 0;
        __syncthreads();
      }
    }
  });
  int other = 0;
  for (int t = 1; t < 1024; ++t) other += took[t] != took[0];
  return took[0] ? other : -1;
}

// Sizes of what a context allocates per job, work item, cell slot and kept deposit.
void sizes(int64_t* out) {
  const int64_t v[] = {sizeof(st::JobDev), sizeof(st::JobAux), sizeof(st::JobPlan), sizeof(st::HistDev),
                       sizeof(st::WorkItem), sizeof(st::CellSlot), st::kRecordBytes};
  std::memcpy(out, v, sizeof(v));
}
int64_t window_cap(int64_t n, int64_t win_deposits) { return st::window_cap(n, win_deposits); }

int keep_bits(const double* edges, int nbins) { return st::keep_bits(edges, nbins); }
int sum_span(int keep_bits, int64_t work) { return st::sum_span(keep_bits, work); }

}  // extern "C"
