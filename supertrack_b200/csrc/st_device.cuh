// Device-side data layout shared by the kernels (vcs_kernels.cu) and the host runtime (capi.cu).
//
// HBM layout of one batch:
//   * input tracks: SoA float64 x, y, z, edep per job (caller memory or the context's arena);
//   * prepared arena (written once per job, read once per oversample): for every job its kept
//     deposits (those that can lie inside the voxel for some shift; in source order, grouped by
//     cell inside each prepare block, or ordered by z layer) as a padded run of warp tiles of kWarpTile deposits.
//     Lane l of a warp tile owns the kDepPerLane consecutive deposits 4l..4l+3 of the tile:
//       PG      : {X, Y} in lattice units, 8 bytes (set_integer_geometry; FP32 variant: float
//                 {x, y}); a lane's four records are one 32-byte load
//       PGZ     : the squared z distance from the layer's centres in the same units (float); a
//                 lane's four are one 16-byte load
//       PSRC    : index of the source deposit in the track, for what is read rarely: deposits that
//                 PG cannot decide, and boundary flags (4 bytes; a track of 2^32 deposits, 128 GB
//                 of x, y, z, edep and 160 GB of records, does not fit the device)
//       PV      : v = edep / ((2/3) d) on the job's fixed-point grid, a 128-bit integer stored
//                 as one 16-byte {low, high} record (one vector load per hit)
//       PKEY    : k_z * N*N (the z part of the sphere key); bit 63 flags boundary deposits
//   * spill tables: one open-addressing table per resident CTA for spheres that do not fit
//     the CTA's shared-memory table (keys, 128-bit accumulators, used-slot list);
//   * histograms: int64 counts and float64 y*f(y) sums per bin, one set per histogram.
#pragma once
#include <math.h>
#include <stdint.h>
#include <cmath>
#include <cstring>
#include "st_core.cuh"

namespace st {

constexpr int64_t kRecordBytes = 8 + 4 + 4 + 16 + 8;  // PG, PGZ, PSRC, PV, PKEY
constexpr int kDepPerLane = 4;                  // deposits owned by one lane inside a warp tile
constexpr int kWarpTile = 32 * kDepPerLane;     // deposits per warp tile
constexpr uint64_t kEmptyKey = ~0ull;           // never a valid sphere key (keys < 2^63)

struct JobDev {
  const double* x;
  const double* y;
  const double* z;
  const double* edep;
  int64_t n;          // deposits in the track
  int64_t n_pad;      // n rounded up to a whole number of warp tiles
  int64_t prep_off;   // first slot of this job in the prepared arena
  double HL;          // scoringRegionHalfLength (after lattice fitting)
  double L;           // scoringRegionLength
  double gSO;         // greatestSphereOffset
  double d;           // sphere diameter
  double inv_d;       // RN(1/d), used by the fast lattice-index path
  double r2;          // RN(r*r)
  double denom;       // RN(RN(2/3)*d): lineal-energy denominator
  double zsh;         // z-origin shift added to every z
  double xy_keep;     // |x|, |y| at or beyond this can never be inside the voxel after a shift
  uint64_t N2;        // N*N
  uint64_t seed;
  uint64_t track_id;
  uint32_t N;
  int32_t n_os;
  int32_t shift_track;
  int32_t hist;       // histogram index
  // boundary flags (see k_prep_flag): computed when `flagged`; the cell hash of the job lives in
  // the cell arena at [cell_off, cell_off + cell_cap); its cells have a side slightly above d (27
  // neighbour cells probed per deposit) or, with cell_nbr8, slightly above 2d (eight probed)
  int32_t flagged;
  uint32_t cell_cap;
  int64_t cell_off;
  double cell_size;
  double inv_cell;    // RN(1 / cell_size)
  // layer windows (see k_prep_write): with `layers` the job may be ordered by z layer; its n_bins bins of
  // 2^bin_shift lattice layers are counted at [bin_off, bin_off + n_bins) of the bin arena, its
  // windows listed from win_off of the window arena
  int64_t bin_off;
  int64_t win_off;
  int32_t layers;
  int32_t n_bins;
  int32_t bin_shift;
  int32_t reserved;
  // FP32 geometry variant: HL', gSO, d, RN(1/d) and r^2 rounded to float (1/d in float)
  float f_HL;
  float f_gSO;
  float f_d;
  float f_inv_d;
  float f_r2;
  int32_t cell_nbr8;
  // integer geometry of the FP64 form (set_integer_geometry)
  double g_scale;     // 2^g_shift / d (0: every deposit is decided in FP64)
  int32_t g_shift;
  int32_t g_ns;       // N 2^g_shift
  float g_lo, g_hi;   // squared distance at or below which a deposit hits, above which it misses
  double wrap_dz;     // |dz| up to which a deposit on a face of the voxel can hit a sphere past the
                      // lattice (set_wrap), -1: none can
};

// Integer geometry: x and y of a deposit and the shift of an oversample in units of d / 2^s, rounded
// to 32-bit integers. The position in the lattice is then V = X + C, with C the shift minus the
// first sphere's centre plus half a cell: its high bits are the sphere index, its low s bits less
// half a cell the offset from the centre, and the deposit is in the voxel when 0 < V < N 2^s.
// X and C are each within 1/2 + 2^-20 unit of the exact value, so V is within 1.25 units. A
// deposit is decided here only if it would be decided the same anywhere in that range: at least 2
// units inside (or outside) the voxel's faces, and a squared distance (in units squared, with the
// z part rounded to float) off the radius by more than `err` below: 2 (2 h 1.25 + 1.25^2) <
// 5 h + 4 from x and y with h = 2^s / 2 the radius, and less than 2^-20 h^2 from four float
// roundings of values near h^2. All others are decided by the FP64 arithmetic, so that hits and
// sphere keys are the reference's bit for bit. N 2^s <= 2^30 keeps every V of a kept deposit
// (|x| < 2HL') inside 32 bits; s <= 22 keeps the offsets exact in float. On a 5,000 nm voxel of
// 2 nm spheres (s = 18) about 3e-5 of the deposits are near enough to a radius to need FP64.
inline void set_integer_geometry(JobDev* D) {
  int s = 22;
  while (s > 0 && ((int64_t)D->N << s) > ((int64_t)1 << 30)) --s;
  const double h = ldexp(0.5, s), err = 5.0 * h + 4.0 + h * h * 0x1p-20;
  D->g_shift = s;
  D->g_ns = (int32_t)((int64_t)D->N << s);
  D->g_scale = ldexp(1.0 / D->d, s);
  D->g_lo = nextafterf((float)(h * h - err), -INFINITY);
  D->g_hi = nextafterf((float)(h * h + err), INFINITY);
  if (!std::isfinite(D->g_scale) || !(D->g_scale >= 0x1p-1000)) {  // d outside the sane range
    D->g_scale = 0.0;
    D->g_lo = -1.0f;
    D->g_hi = INFINITY;
  }
}

// Keys of spheres past the lattice. A deposit within a rounding of a face of the voxel can round to
// lattice index N (or -1), one past the lattice, and hit there when it lies on that sphere's axis.
// The key of (kx, N, kz) is that of (kx, 0, kz + 1): the reference sums the two as one sphere, although
// they are a voxel apart, so a job with such a deposit must not be cut into windows. set_wrap finds
// whether the lattice's roundings allow it and for which z; may_wrap then asks for a deposit with such
// a z whether some shift (24 bits) puts its x or y there, both in the reference's arithmetic. (The FP32
// variant's floats wrap at other values, which are not looked for.)
struct WrapLattice {
  double HL, L, gSO, d, r2;
  uint32_t N;
};
// Whether coordinate c (after the shift) is in the voxel, past the lattice, and within r of that sphere.
ST_HD bool wraps(const WrapLattice& g, double c, double* dc) {
  if (!(fabs(c) < g.HL)) return false;
  const double a = st_dsub(c, g.gSO);
  const double k = rint(a / g.d);
  *dc = st_dsub(st_dmul(k, g.d), a);
  return (k < 0.0 || k >= (double)g.N) && st_dmul(*dc, *dc) <= g.r2;
}
ST_HD bool may_wrap(const WrapLattice& g, int shift_track, double c) {
  double dc;
  if (!shift_track) return wraps(g, st_dadd(c, shift_from_uniform(0.5f, g.L, g.HL)), &dc);
  bool any = false;
  for (int face = -1; face <= 1; face += 2) {
    const double m = rint((face * g.HL - c + g.HL) / g.L * 0x1p24);  // the uniform that puts c there
    for (int k = -2; k <= 2; ++k) {
      const double u = (m + k) * 0x1p-24;
      if (u > 0.0 && u <= 1.0)
        any |= wraps(g, st_dadd(c, shift_from_uniform((float)u, g.L, g.HL)), &dc);
    }
  }
  return any;
}
inline void set_wrap(JobDev* D) {
  const WrapLattice g = {D->HL, D->L, D->gSO, D->d, D->r2, D->N};
  D->wrap_dz = -1.0;
  if (!D->flagged) return;
  for (int face = -1; face <= 1; face += 2) {  // (farther from the face leaves less for dz)
    double dc;
    if (wraps(g, face * std::nextafter(D->HL, 0.0), &dc))
      D->wrap_dz = std::fmax(D->wrap_dz, std::sqrt(g.r2 * (1.0 + 0x1p-50) - dc * dc));
  }
}

// Deposits of a windowed job are processed in windows of consecutive kept deposits: kWindow (two
// warp tiles per warp of the fused kernel's CTA), or twice that for jobs with coarse windows. A
// kept deposit is a boundary deposit when a kept deposit of another window lies within distance d
// of it; the flag travels in bit 63 of its PKEY word (keys are below 2^63).
constexpr unsigned long long kBoundaryBit = 1ull << 63;

// How a job's oversamples are cut into windows that empty the sphere table (JobAux::windowed):
// not at all, windows of the source order with boundary flags, or windows of whole z layers.
constexpr int kWinNone = 0;
constexpr int kWinFlags = 1;
constexpr int kWinLayers = 2;
constexpr int kMaxBins = 4096;                        // z bins of a layered job
constexpr unsigned long long kWinContinues = 1ull << 63;  // window list: the bin began earlier
// Most entries of a job's window list: two consecutive windows hold more than one window's
// deposits, a bin larger than a window ends with a short one, plus the closing entry.
constexpr int64_t window_cap(int64_t n, int64_t win_deposits) { return 3 * (n / win_deposits) + 8; }

// z bins of a layered job: one per lattice layer, or per 2^bin_shift layers on a lattice of more
// than kMaxBins.
inline int bin_shift(uint32_t N) {
  int s = 0;
  while (((N - 1) >> s) >= (uint32_t)kMaxBins) ++s;
  return s;
}
inline int bin_count(uint32_t N) { return (int)((N - 1) >> bin_shift(N)) + 1; }

// Per-job values produced on the device.
struct JobAux {
  int32_t e_min;          // min ulp exponent over nonzero contributions
  int32_t e_max;          // max ulp exponent over nonzero contributions
  int32_t flags;          // kAuxNonzero | kAuxNonfinite
  int32_t windowed;       // set by k_prep_scan: kWinNone, kWinFlags (JobDev::flagged and more
                          // than PrepareParams::flag_min_kept kept deposits) or kWinLayers
  long long kept;              // deposits that can be inside the voxel for some shift
  unsigned long long hits;     // in-sphere deposits summed over all oversamples
  unsigned long long spheres;  // (oversample, sphere) pairs with at least one hit
  unsigned long long binned;   // of those, the ones that landed inside the histogram range
  unsigned long long inbox;    // deposit*oversamples inside the voxel after the shift
  unsigned long long cells;    // occupied cells: of the boundary-flag hash (kWinFlags), or of
                               // each prepare block, summed (kWinLayers)
  int32_t n_win;               // windows of a layered job
  int32_t reserved;
};
constexpr int kAuxNonzero = 1;
constexpr int kAuxNonfinite = 2;
constexpr int kAuxWraps = 4;  // some shift can put a deposit past the lattice (may_wrap)

struct HistDev {
  const double* edges;            // nbins + 1 edges
  unsigned long long* counts;     // nbins
  double* yfy;                    // nbins
  int32_t nbins;
  int32_t mode;                   // bin guess: 0 linear in y, 1 linear in log2(y)
  double ca, cb;                  // guess = (y - ca) * cb  or  (log2(y) - ca) * cb
  int32_t keep_bits;              // a CTA keeps the histogram for 2^keep_bits deposit*oversamples
  int32_t reserved;
};

// A CTA's copy of a histogram holds the y*f(y) sum of a bin as a signed 128-bit integer in units of
// the lower edge's last place. A y of 2^up times the edge or more (up: the difference of the
// exponents) has 53 + up bits and 2^k of them have 53 + up + k, which must stay below 127: kSumBits
// bits are left for up and k. The copy is kept for at most 2^31 deposit*oversamples (32-bit counts),
// fewer if the widest bin needs the room, down to the 2^18 of one large work item; a y that is too
// far above its edge even then is added to HBM as a double (sum_span).
constexpr int kSumBits = 126 - 53;
inline int keep_bits(const double* edges, int nbins) {
  const auto exponent = [&](int b) {  // biased; 0 and below: not a positive normal number
    int64_t bits;
    std::memcpy(&bits, &edges[b], 8);
    return (int)(bits >> 52);
  };
  int first = 0;
  while (first < nbins && exponent(first) <= 0) ++first;
  int span = exponent(nbins) - exponent(first);  // of all such bins: usually little enough
  if (kSumBits - span < 31) {
    span = 0;
    for (int b = first; b < nbins; ++b) {
      const int s = exponent(b + 1) - exponent(b);
      span = s > span ? s : span;
    }
  }
  const int k = kSumBits - span;
  return k < 18 ? 18 : (k > 31 ? 31 : k);
}

// Largest difference of exponents between a y and its bin's lower edge at which the 128-bit sum
// takes it, in a copy kept for 2^keep_bits deposit*oversamples or for one item of more (`work`).
ST_HD int sum_span(int keep_bits, long long work) {
  const int w = work > 1 ? 64 - clz64((uint64_t)(work - 1)) : 0;  // work <= 2^w
  return kSumBits - (w > keep_bits ? w : keep_bits);
}

// One unit of work for the persistent kernel: a contiguous block of oversamples of one job, or part
// of one oversample. A batch has room for total oversamples * max_helpers of them: 16 bytes.
struct WorkItem {
  int32_t job;
  int32_t os_begin;
  int32_t os_count;   // negative: part of oversample os_begin of a layered job, -os_count windows
  int32_t unit;       // >= 0: a helper of shared unit `unit` (one oversample of a large job, split
                      // into chunks); -1: the CTA does every window of its oversamples; -1 - p:
                      // part p of the oversample
};

// One exported sphere: (oversample, key, lineal energy, hit deposits).
struct SphereRecord {
  uint64_t key;
  double y;
  int32_t os;
  int32_t job;
};

struct FusedParams {
  const JobDev* jobs;
  JobAux* aux;
  const HistDev* hists;
  const WorkItem* items;
  const int* n_items;         // written by the planner
  int32_t flush_threshold;    // smem table occupancy that triggers a flush to the spill table
  unsigned int* work_counter; // next item to claim
  const int2* PG;             // {X, Y} in lattice units (FP32 variant: float2 {x, y})
  const float* PGZ;           // squared z distance, in lattice units (FP32 variant: nm)
  const uint32_t* PSRC;       // index in the track, for deposits that PG cannot decide
  const ulonglong2* PV;            // contribution on the job's grid: {low, high} 64-bit words
  const unsigned long long* PKEY;  // k_z * N*N, bit 63 = boundary deposit
  // spill tables: gridDim.x tables of gcap slots each
  uint64_t* gkeys;
  unsigned long long* glo;
  unsigned long long* ghi;
  uint32_t* gused;
  unsigned int* gcount;       // gridDim.x counters
  uint32_t gcap;              // power of two
  int32_t smem_hist_bins;     // histograms with more bins accumulate straight into HBM
  // optional export of every sphere (os, key, y); null when not requested
  SphereRecord* export_buf;
  unsigned long long* export_count;
  unsigned long long export_cap;
  int* error_flags;           // bit 0: spill table full, bit 1: export buffer full,
                              // bit 2: spill-table pool exhausted, bit 3: unit wait gave up
  // shared units (one oversample of a large job, processed in chunks by several CTAs)
  unsigned int* unit_next;    // next chunk to claim
  unsigned int* unit_done;    // chunks finished
  int* unit_table;            // spill table of the unit (-1 none yet, -2 being acquired)
  unsigned int* pool_bits;    // spill tables in use (one bit per table, gridDim.x tables)
  const unsigned long long* wins;  // window lists of layered jobs (first kept deposit of each)
  int32_t chunk_windows;      // windows per chunk
  int32_t fp32;               // 1: FP32 geometry variant (float records, float x/y geometry)
};

// One slot of the cell hash used for boundary flags: the cell key (EMPTY when free), the
// smallest window with a deposit in the cell and the bitwise complement of the largest one, so
// that an all-ones fill is the empty state and both bounds are kept with atomicMin. One 16-byte
// load reads a whole slot.
struct __align__(16) CellSlot {
  unsigned long long key;
  unsigned int wmin;
  unsigned int nwmax;
};

struct PrepareParams {
  const JobDev* jobs;
  JobAux* aux;
  int32_t n_jobs;
  int64_t blk_base;           // prepare block of blockIdx.x 0 (jobs and blk_prefix may start
                              // at a later job of the batch; block indices stay batch-wide)
  const int64_t* blk_prefix;  // n_jobs+1 prefix sums of prepare blocks per job
  const int32_t* blk_job;     // batch-wide job index of each prepare block (null: searched in
                              // blk_prefix)
  int32_t job_base;           // batch-wide index of jobs[0]
  int32_t* blk_count;         // kept deposits per prepare block
  int64_t* blk_offset;        // first kept index of each prepare block inside its job
  CellSlot* cells;            // cell arena (flagged jobs)
  uint32_t* bins;             // z bins of layered jobs: kept deposits, then first free place
  unsigned long long* wins;   // window lists of layered jobs
  int32_t win_tiles;          // warp tiles of a layer window (twice that on dense tracks)
  int64_t cta_share;          // deposit*oversamples of the launch per CTA of the fused kernel
  int64_t unit_min;           // kept deposits above which an oversample of a job with boundary flags
                              // is spread over CTAs (a shared unit)
  int32_t* any_flags;         // set when a job of the launch runs with window boundary flags
  int2* PG;                   // records as in FusedParams
  float* PGZ;
  uint32_t* PSRC;
  ulonglong2* PV;
  unsigned long long* PKEY;
  int32_t fp32;               // 1: records for the FP32 geometry variant
  int64_t flag_min_kept;      // a flagged job runs with window flags only above this many kept
                              // deposits (fewer spheres than that fit the table without them)
  int32_t sort;               // prepare blocks that write their kept deposits grouped by cell
                              // (see k_prep_write): 0 none, 1 those of window-flagged jobs,
                              // 2 all; the others write them in source order
};

// Device-side planning of the fused kernel's work items from the kept deposit counts.
constexpr int kMaxHelpers = 32;  // default of JobPlan's helpers per unit and parts per oversample
constexpr int kPlanBuckets = 64;
struct JobPlan {
  int32_t items;
  int32_t bucket;
  int32_t unit_base;   // -1: private items
  int32_t blk_os;      // oversamples per private item, or helpers per unit
  int32_t blk_win;     // windows per item of a job whose oversamples are split into parts, else 0
};
struct PlanParams {
  const JobDev* jobs;
  const JobAux* aux;
  int32_t n_jobs;
  int32_t chunk_windows;
  int32_t max_helpers;
  int32_t grid;
  long long item_cost;
  int32_t share_divisor;             // a job is shared when kept > total / (share_divisor * grid)
  int32_t min_chunks;                // ... and kept > min_chunks chunks; share_divisor 0: never
  unsigned int* bucket_start;        // kPlanBuckets
  unsigned int* bucket_cursor;       // kPlanBuckets
  unsigned int* unit_counter;
  JobPlan* plan;
  WorkItem* items;
  int* n_items;
  long long item_cap;
};

// A run's state on the device that starts from fixed values, set by one kernel (launch_reset).
struct ResetParams {
  JobAux* aux;                 // n_jobs job records: exponent range empty, everything else zero
  int32_t n_jobs;
  int32_t n_pool;
  unsigned int* counter;       // 4 words of zeros: work counter, any_flags
  unsigned int* pool;          // n_pool words of zeros
  unsigned int* plan;          // the planner's scratch, kPlanScratch bytes of zeros
  unsigned int* u_next;        // n_units words each: zeros, zeros, all ones
  unsigned int* u_done;
  unsigned int* u_table;
  int64_t n_units;
  uint32_t* bins;              // n_bins words of zeros
  int64_t n_bins;
  unsigned int* err;           // 4 words of zeros (null: kept)
  unsigned int* ex_count;      // 4 words of zeros (null: none)
  // empty spill tables (null: kept): n_slots keys of ones and sums of zeros, n_tables counters
  uint64_t* gkeys;
  unsigned long long* glo;
  unsigned long long* ghi;
  unsigned int* gcount;
  int64_t n_slots;
  int32_t n_tables;
};
// the planner's scratch: item count, unit counter, buckets' starts and cursors, in bytes
constexpr int kPlanScratch = 8 + 2 * 4 * kPlanBuckets;

constexpr int kPrepThreads = 256;
constexpr int kPrepSlotsPerBlock = 1024;                // source deposits per prepare block
constexpr int kFusedWarps = 32;                       // warps of the fused kernel's CTA
constexpr int kCtaTile = kFusedWarps * kWarpTile;    // kept deposits of one warp tile per warp
constexpr int kWinTiles = 2;                          // warp tiles per warp in a window
constexpr int kCoarseTiles = 4;                       // ... in a coarse window (dense spheres)
constexpr int kWindow = kWinTiles * kCtaTile;         // kept deposits per window (8192)
// Warp tiles of a shared unit's chunk: chunk_windows windows of kWinTiles tiles per warp,
// rounded up to whole coarse windows, so that no window is ever split between two chunks.
ST_HD int64_t chunk_tiles(int chunk_windows) {
  constexpr int64_t kCoarse = (int64_t)kFusedWarps * kCoarseTiles;
  const int64_t t = (int64_t)chunk_windows * kFusedWarps * kWinTiles;
  return (t + kCoarse - 1) / kCoarse * kCoarse;
}

// A flagged job uses flag cells of side 2d (eight probes per deposit instead of 27, but more
// deposits flagged, whose spheres then pass through the spill log at every oversample) when its
// deposits per sphere diameter of track length, n * d / (2 HL), times its oversamples are at most
// this (context parameter flag_cells_limit).
constexpr int64_t kFlagCellsLimit = 25000;
constexpr int kCellBits = 21;                         // bits per axis of a cell key

// A job qualifies for windows (JobDev::flagged): several of them, on a fine lattice, for several
// oversamples.
inline bool job_flagged(int64_t n, int64_t n_os, uint32_t N) {
  return n > 2 * kCtaTile && n_os >= 4 && N >= 128 && N < (1u << (kCellBits - 2));
}

// Device bytes that one job of a batch takes in a context's arrays: its track (x, y, z, edep), the
// prepared records, the cell hash, z bins and window list of a job that qualifies for windows, its tables, prepare blocks, work items and units, and one histogram of its own. The
// server admits jobs by it, so it must not be less than what build_tables allocates per job.
inline int64_t job_device_bytes(int64_t n, int64_t n_os, uint32_t N, int nbins, int max_helpers) {
  const int64_t n_pad = ((n > 1 ? n : 1) + 255) / 256 * 256;
  const int64_t blocks = (n_pad + kPrepSlotsPerBlock - 1) / kPrepSlotsPerBlock;
  int64_t b = 32 * n + kRecordBytes * n_pad;
  if (job_flagged(n, n_os, N)) {
    int64_t cells = 1;
    while (cells < 2 * n) cells <<= 1;
    b += cells * (int64_t)sizeof(CellSlot);
    b += 4 * (int64_t)bin_count(N) + 8 * window_cap(n, kCtaTile);
  }
  b += (int64_t)(sizeof(JobDev) + sizeof(JobAux) + sizeof(JobPlan) + sizeof(HistDev)) + 8 + 16 * blocks;
  b += n_os * (max_helpers * (int64_t)sizeof(WorkItem) + 12);
  return b + 16 * (int64_t)nbins + 8 * ((int64_t)nbins + 1);
}

}  // namespace st
