// sm_100a kernels of the VoxelConstrainedSphere superimposition path.
//
//   prepare   : once per run of a track (k_prep_*). z-origin shift, the deposits that
//               can be in the voxel for some shift, x and y in lattice units, the z part of the
//               lattice test (k_z and (k_z*d - a_z)^2, which do not depend on the oversample), the
//               lineal energy contribution v = edep/((2/3)d), the job's fixed-point exponent range,
//               and the compaction of the kept deposits into the prepared arena.
//               Follows VoxelConstrainedSphereMethod.cu:138-154 (z shift), :198 (|z| test),
//               :249-258 (z axis of the membership test), :302/:322 (lineal denominator).
//   k_fused   : persistent work-stealing kernel over (job, oversample block) items. Per
//               oversample: Philox shift, x/y shift + strict box test (:176-198), x/y lattice
//               indices and the inclusive sphere test (:249-271), the 64-bit key (:313-318),
//               exact reduce-by-key of the contributions (Histogram.cu:150-153) in registers,
//               shared memory and, when a job's spheres overflow shared memory, the CTA's spill
//               table in HBM, and the HistogramRange binning of each sphere's lineal energy
//               (Histogram.cu:158) plus its y*f(y) weight, accumulated over oversamples
//               (Histogram.cu:161-171).
#include <cuda_runtime.h>
#include <limits.h>
#include "planning.cuh"
#include "st_device.cuh"

namespace st {

__device__ __forceinline__ uint32_t slot_hash(uint64_t key, uint32_t mask) {
  return (uint32_t)((key * 0x9E3779B97F4A7C15ull) >> 40) & mask;
}

// Slot of a sphere key in the shared-memory table: Fibonacci hashing proper, the top
// log2(mask + 1) bits of key * 2^64/phi (mask + 1 a power of two of at least 2). The middle bits
// that slot_hash takes map the regular lattice keys of a straight track into long runs of
// neighbouring slots, which at a quarter load already exceeded the 32-slot probe limit.
__device__ __forceinline__ uint32_t table_hash(uint64_t key, uint32_t mask) {
  return (uint32_t)((key * 0x9E3779B97F4A7C15ull) >> 32) >> __clz((int)mask);
}

// ---------------------------------------------------------------------------------------------
// Lattice index along one axis, k = llrint(a / d), bit-exact with the IEEE quotient. The fused
// kernel forms q = RN(a * RN(1/d)), whose distance to RN(a/d) is below |q| * 2^-51.2; it takes
// k = rint(q) (adding and subtracting 1.5 * 2^52 rounds to the nearest integer, ties to even)
// unless q lies within 2^-20 of a half-integer, where the correctly rounded division decides.
// ---------------------------------------------------------------------------------------------
constexpr double kMagic = 0x1.8p52;             // adding it rounds |q| < 2^51 to an integer
constexpr double kRiskBand = 0.5 - 0x1p-20;     // |q - rint(q)| at or above it: decide exactly

// The same, for one value: k = llrint(a / d) for |a / d| < 2^21.
__device__ __forceinline__ double lattice_index(double a, double d, double inv_d) {
  const double q = st_dmul(a, inv_d);
  const double k = st_dsub(st_dadd(q, kMagic), kMagic);
  return fabs(st_dsub(q, k)) >= kRiskBand ? rint(__ddiv_rn(a, d)) : k;
}

// ---------------------------------------------------------------------------------------------
// Prepare stage (once per run of a track): four launches, six when a job may run with boundary flags.
//   k_prep_count : per block of kPrepSlotsPerBlock source deposits, the number of deposits that
//                  can lie inside the voxel for some oversample (z after the z-origin shift
//                  strictly inside; |x|, |y| below xy_keep), plus the job's exponent range of
//                  the contributions v = edep/((2/3)d) over all its deposits, and the z bins of
//                  jobs that qualify for layer windows;
//   k_prep_scan  : per job, exclusive scan of its block counts -> block offsets, kept total, window
//                  mode (planning.cuh);
//   k_prep_cells : empties the cell hashes of jobs with boundary flags;
//   k_prep_write : compaction of the kept deposits into the prepared arena (source order, grouped
//                  by cell, or by z layer) with the oversample-independent z part of the lattice
//                  test, and the cells of jobs with boundary flags;
//   k_prep_pad   : padding of each job's last warp tile (outside the voxel for every shift), and the
//                  window lists of layered jobs;
//   k_prep_flag  : the boundary flags.
// A dropped deposit can be inside the box for no shift, so dropping it changes no result.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ int find_job(const int64_t* blk_prefix, int n_jobs, int64_t b) {
  int lo = 0, hi = n_jobs;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (blk_prefix[mid] <= b) lo = mid; else hi = mid;
  }
  return lo;
}

// The job of prepare block b: one load from the block table, which saves the short prepare
// blocks a dozen dependent loads of the binary search before their first track load.
__device__ __forceinline__ int prep_job(const PrepareParams& p, int64_t b) {
  return p.blk_job ? __ldg(&p.blk_job[b]) - p.job_base : find_job(p.blk_prefix, p.n_jobs, b);
}

// Slot of kept deposit k of a job in the prepared arena.
__device__ __forceinline__ int64_t prep_slot(const JobDev& J, int64_t k) { return J.prep_off + k; }

// z bin of a kept deposit (z after the z-origin shift): its lattice layer k_z, clamped to the
// lattice (k_z can round to -1 or N on the voxel's faces), over 2^bin_shift.
__device__ __forceinline__ int z_bin(const JobDev& J, double z1) {
  const int k = (int)lattice_index(st_dsub(z1, J.gSO), J.d, J.inv_d);
  return min(max(k, 0), (int)J.N - 1) >> J.bin_shift;
}

__device__ __forceinline__ bool keep_deposit(const JobDev& J, double x, double y, double z) {
  const double z1 = st_dadd(z, J.zsh);
  return fabs(z1) < J.HL && fabs(x) < J.xy_keep && fabs(y) < J.xy_keep;
}

// Flag cell of side cell_size containing (x, y, z): integer cell coordinates, offset to be
// non-negative, from u = RN(c * RN(1/cell_size)) per axis (within |u| 2^-51 of the exact
// quotient, below 2^-31 for the coordinates of a flagged job, |u| < 2^20). A job's flag cells
// have a side slightly above d or slightly above 2d (JobDev::cell_nbr8). With side d, two
// deposits within distance d of each other lie in the same or in adjacent cells: 27 cells around
// a point hold every deposit within d of it. With side 2d, a deposit within d of a point lies in
// the point's cell or in the neighbour cell on the side of the half of the cell the point is in:
// per axis, |u' - u| < 1/2 - 2^-12 for the other deposit's u', so floor(u') is floor(u) - 1 or
// floor(u) when u - floor(u) < 1/2, and floor(u) or floor(u) + 1 otherwise (the rounding errors
// are far below the margin): eight cells hold every deposit within d.
struct CellCoord {
  long long x, y, z;
};

__device__ __forceinline__ CellCoord cell_of(double x, double y, double z, double inv_cs) {
  const long long off = 1ll << (kCellBits - 1);
  return {(long long)floor(st_dmul(x, inv_cs)) + off, (long long)floor(st_dmul(y, inv_cs)) + off,
          (long long)floor(st_dmul(z, inv_cs)) + off};
}

// The cell of a point (as cell_of) and, per axis, the side of its neighbour cells (-1: the point
// is in the lower half of its cell).
struct CellNbr {
  CellCoord c;
  int sx, sy, sz;
};

__device__ __forceinline__ int half_side(double u) {
  return st_dsub(u, floor(u)) < 0.5 ? -1 : 1;
}

__device__ __forceinline__ CellNbr cell_nbr(double x, double y, double z, double inv_cs) {
  const long long off = 1ll << (kCellBits - 1);
  const double u = st_dmul(x, inv_cs), v = st_dmul(y, inv_cs), w = st_dmul(z, inv_cs);
  return {{(long long)floor(u) + off, (long long)floor(v) + off, (long long)floor(w) + off},
          half_side(u), half_side(v), half_side(w)};
}

// Key of the cell at offset (dx, dy, dz) from c.
__device__ __forceinline__ uint64_t cell_key(const CellCoord& c, int dx, int dy, int dz) {
  return ((uint64_t)(c.z + dz) << (2 * kCellBits)) | ((uint64_t)(c.y + dy) << kCellBits) |
         (uint64_t)(c.x + dx);
}

// Records window `win` in the cell `key`; true when this call created the cell.
__device__ __forceinline__ bool cell_insert(const PrepareParams& p, const JobDev& J,
                                            uint64_t key, uint32_t win) {
  const uint32_t mask = J.cell_cap - 1;
  uint32_t h = slot_hash(key, mask);
  for (uint32_t probe = 0; probe < J.cell_cap; ++probe) {
    CellSlot* slot = p.cells + J.cell_off + h;
    const uint64_t k = __ldcg(&slot->key);
    bool mine = k == key, created = false;
    if (!mine && k == kEmptyKey) {
      const uint64_t old = atomicCAS(&slot->key, kEmptyKey, key);
      created = old == kEmptyKey;
      mine = created || old == key;
    }
    if (mine) {
      atomicMin(&slot->wmin, win);
      atomicMin(&slot->nwmax, ~win);
      return created;
    }
    h = (h + 1) & mask;
  }
  return false;
}

// True when the cell slot v holds a deposit of a window other than `win`; windows are compared
// after a right shift by `shift` (1: coarse windows of two recorded windows each).
__device__ __forceinline__ bool slot_foreign(const ulonglong2& v, uint32_t win, int shift) {
  return ((uint32_t)v.y >> shift) != (win >> shift) ||
         (~(uint32_t)(v.y >> 32) >> shift) != (win >> shift);
}

// Neighbour keys as offsets from a cell's key: the coordinate fields of every cell a flagged job
// probes stay inside [0, 2^kCellBits), so a key of the cell at (dx, dy, dz) from c is c's key plus
// dz 2^(2 kCellBits) + dy 2^kCellBits + dx in two's complement. Neighbour c (0..26) of the 27
// around a side-d cell has (c % 3 - 1, c / 3 % 3 - 1, c / 9 - 1); neighbour c (0..7) of the eight
// around a point in a side-2d cell adds n.sx on x when bit 0 of c is set, n.sy on y for bit 1 and
// n.sz on z for bit 2.
__host__ __device__ constexpr int64_t cell_offset(int dx, int dy, int dz) {
  return (int64_t)dz * ((int64_t)1 << (2 * kCellBits)) + (int64_t)dy * ((int64_t)1 << kCellBits) + dx;
}
__device__ __forceinline__ uint64_t nbr_key27(uint64_t base, int c) {
  return base + (uint64_t)cell_offset(c % 3 - 1, (c / 3) % 3 - 1, c / 9 - 1);
}
struct NbrOffsets {
  uint64_t base;
  int64_t ox, oy, oz;
};
__device__ __forceinline__ NbrOffsets nbr_offsets8(const CellNbr& n) {
  return {cell_key(n.c, 0, 0, 0), cell_offset(n.sx, 0, 0), cell_offset(0, n.sy, 0),
          cell_offset(0, 0, n.sz)};
}
__device__ __forceinline__ uint64_t nbr_key8(const NbrOffsets& o, int c) {
  return o.base + (uint64_t)(((c & 1) ? o.ox : 0) + ((c & 2) ? o.oy : 0) + ((c & 4) ? o.oz : 0));
}

// True when one of the neighbour cells c0 .. c0 + BATCH - 1 (keys from key_of) holds a deposit
// of another window. Their first hash slots are loaded together, so a lane has several L2
// round trips in flight instead of one; a cell whose first slot holds another key continues
// probing alone. The neighbourhoods of a block's deposits overlap, so cached loads serve many probes
// from L1; plain ones, since k_prep_write may still fill the hash when this kernel is launched
// (the non-coherent path is for what stays as it is while the kernel lives).
template <int BATCH, typename KeyOf>
__device__ __forceinline__ bool cells_foreign(const PrepareParams& p, const JobDev& J,
                                              const KeyOf& key_of, int c0, uint32_t win,
                                              int shift) {
  const uint32_t mask = J.cell_cap - 1;
  const CellSlot* base = p.cells + J.cell_off;
  ulonglong2 v[BATCH];
  uint32_t h[BATCH];
#pragma unroll
  for (int t = 0; t < BATCH; ++t) {
    h[t] = slot_hash(key_of(c0 + t), mask);
    v[t] = *reinterpret_cast<const ulonglong2*>(base + h[t]);
  }
  bool foreign = false;
#pragma unroll
  for (int t = 0; t < BATCH; ++t) {
    const uint64_t key = key_of(c0 + t);
    if (v[t].x == key) {
      foreign |= slot_foreign(v[t], win, shift);
    } else if (v[t].x != kEmptyKey) {
      uint32_t hh = h[t];
#pragma unroll 1
      for (uint32_t probe = 1; probe < J.cell_cap; ++probe) {
        hh = (hh + 1) & mask;
        const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(base + hh);
        if (w.x == key) {
          foreign |= slot_foreign(w, win, shift);
          break;
        }
        if (w.x == kEmptyKey) break;
        if (probe == J.cell_cap - 1) foreign = true;  // a full table: conservative
      }
    }
  }
  return foreign;
}

// The z bins that a prepare block meets, in shared memory: the block adds to a bin's word in HBM once
// instead of once per warp or cell group, which on tracks across z all meet on a few words (prepare
// of one track of 4e6 deposits, 10 nm, across z 0.69 -> 0.27 ms, along z 0.39 -> 0.23). A bin that finds its
// place taken four times goes to HBM directly; a block of many bins is no contention, nor are the few
// blocks of a job of up to kGatherMin deposits (one proton track of 19,997: 1.5 us saved).
constexpr int kBlockBins = 64;
constexpr int64_t kGatherMin = 64 * kPrepSlotsPerBlock;
__device__ __forceinline__ int block_bin(int* keys, int bin) {
  int h = bin & (kBlockBins - 1);
#pragma unroll 1
  for (int probe = 0; probe < 4; ++probe) {
    int k = *(volatile int*)&keys[h];
    if (k < 0) {
      k = atomicCAS(&keys[h], -1, bin);
      if (k < 0) k = bin;
    }
    if (k == bin) return h;
    h = (h + 1) & (kBlockBins - 1);
  }
  return -1;
}

// Distance of z (as submitted) from the centre plane of its layer.
__device__ __forceinline__ double layer_dz(const JobDev& J, double z) {
  const double az = st_dsub(st_dadd(z, J.zsh), J.gSO);
  return fabs(st_dsub(st_dmul(lattice_index(az, J.d, J.inv_d), J.d), az));
}

// Eight blocks per SM (32 registers): more track loads in flight.
__global__ void __launch_bounds__(kPrepThreads, 8) k_prep_count(PrepareParams p) {
  chain_start();
  const int64_t b = p.blk_base + blockIdx.x;
  const int j = prep_job(p, b);
  const JobDev J = p.jobs[j];
  const int64_t i0 = (b - p.blk_prefix[j]) * (int64_t)kPrepSlotsPerBlock;
  int emin = INT_MAX, emax = INT_MIN, flags = 0, kept = 0;
  bool on_plane = false;  // some deposit so close to the centre plane of its layer that it might wrap
  __shared__ int s_key[kBlockBins];
  __shared__ unsigned s_count[kBlockBins];
  const bool gather = J.layers && J.n > kGatherMin;
  if (gather) {
    if (threadIdx.x < kBlockBins) {
      s_key[threadIdx.x] = -1;
      s_count[threadIdx.x] = 0;
    }
    __syncthreads();
  }
  // a guard rather than a break, so that the loads of all rounds can be in flight together
#pragma unroll
  for (int s = threadIdx.x; s < kPrepSlotsPerBlock; s += kPrepThreads) {
    const int64_t i = i0 + s;
    const bool in = i < J.n;
    const double z = in ? J.z[i] : 0.0;
    const bool keep = in && keep_deposit(J, J.x[i], J.y[i], z);
    kept += keep ? 1 : 0;
    if (J.flagged) on_plane |= keep && layer_dz(J, z) <= J.wrap_dz;
    if (J.layers) {
      // neighbouring deposits lie in few layers: one addition per layer and warp (one per deposit
      // met on the same words: 7.9 ms instead of about 1.6 for 32e6 deposits of 10 nm ion tracks)
      const int bin = keep ? z_bin(J, st_dadd(z, J.zsh)) : -1;
      const unsigned same = __match_any_sync(0xffffffffu, bin);
      if (keep && (int)(threadIdx.x & 31) == __ffs(same) - 1) {
        const int q = gather ? block_bin(s_key, bin) : -1;
        atomicAdd(q >= 0 ? &s_count[q] : &p.bins[J.bin_off + bin], (unsigned)__popc(same));
      }
    }
    if (!in) continue;
    const double v = __ddiv_rn(J.edep[i], J.denom);
    if (!isfinite(v)) {
      flags |= kAuxNonfinite;
    } else if (v != 0.0) {
      flags |= kAuxNonzero;
      const int ex = ulp_exponent(v);
      emin = min(emin, ex);
      emax = max(emax, ex);
    }
  }
  if (on_plane) {
    const WrapLattice g = {J.HL, J.L, J.gSO, J.d, J.r2, J.N};
#pragma unroll 1
    for (int64_t i = i0 + threadIdx.x; i < J.n && i < i0 + kPrepSlotsPerBlock; i += kPrepThreads)
      if (layer_dz(J, J.z[i]) <= J.wrap_dz && keep_deposit(J, J.x[i], J.y[i], J.z[i]) &&
          (may_wrap(g, J.shift_track, J.x[i]) || may_wrap(g, J.shift_track, J.y[i])))
        flags |= kAuxWraps;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    emin = min(emin, __shfl_xor_sync(0xffffffffu, emin, o));
    emax = max(emax, __shfl_xor_sync(0xffffffffu, emax, o));
    flags |= __shfl_xor_sync(0xffffffffu, flags, o);
    kept += __shfl_xor_sync(0xffffffffu, kept, o);
  }
  // the block's warps meet in shared memory; one thread updates the job's record, whose
  // address every block of the job shares
  __shared__ int s_kept, s_flags, s_emin, s_emax;
  if (threadIdx.x == 0) {
    s_kept = 0;
    s_flags = 0;
    s_emin = INT_MAX;
    s_emax = INT_MIN;
  }
  __syncthreads();
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&s_kept, kept);
    if (flags) {
      atomicOr(&s_flags, flags);
      atomicMin(&s_emin, emin);
      atomicMax(&s_emax, emax);
    }
  }
  __syncthreads();
  if (gather && threadIdx.x < kBlockBins && s_count[threadIdx.x])
    atomicAdd(&p.bins[J.bin_off + s_key[threadIdx.x]], s_count[threadIdx.x]);
  if (threadIdx.x == 0) {
    p.blk_count[b] = s_kept;
    if (s_flags) {
      atomicOr(&p.aux[j].flags, s_flags);
      if (s_flags & kAuxNonzero) {
        atomicMin(&p.aux[j].e_min, s_emin);
        atomicMax(&p.aux[j].e_max, s_emax);
      }
    }
  }
}

// Empties the cell hash of every job that runs with window boundary flags (all-ones is the empty
// slot); any number of CTAs.
__global__ void __launch_bounds__(kPrepThreads) k_prep_cells(PrepareParams p) {
  chain_start();
  if (!*p.any_flags) return;
  __shared__ int s_jobs[kPrepThreads];
  __shared__ int s_n;
  for (int base = 0; base < p.n_jobs; base += kPrepThreads) {
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
    const int j = base + threadIdx.x;
    if (j < p.n_jobs && p.aux[j].windowed == kWinFlags) s_jobs[atomicAdd(&s_n, 1)] = j;
    __syncthreads();
    for (int q = 0; q < s_n; ++q) {
      const JobDev& J = p.jobs[s_jobs[q]];
      uint4* slots = reinterpret_cast<uint4*>(p.cells + J.cell_off);
      for (uint32_t i = blockIdx.x * kPrepThreads + threadIdx.x; i < J.cell_cap; i += gridDim.x * kPrepThreads)
        slots[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
    }
    __syncthreads();
  }
}

// In-block grouping of kept deposits by cell (sorted prepare blocks): a block writes its kept
// deposits grouped by d-cell (x, y and z after the z-origin shift, each divided by d and rounded
// down), the groups in the order of their cells' first deposit in the block. Deposits of one cell
// mostly share a sphere for any shift, so the fused kernel sums them as runs in registers and
// across lanes instead of one shared-memory insert each; line-ordered tracks keep their order
// apart from the deposits pulled forward to their cell's first one. Cells are told apart by a
// kCellHashBins-way hash (a collision only merges two groups). Sort mode 1 groups the blocks of
// window-flagged jobs (multi-window jobs on fine lattices: the dense tracks whose spheres take
// several hits that the source order scatters), mode 2 every block.
constexpr int kCellHashBins = 1024;
__device__ __forceinline__ unsigned cell_hash_bin(const JobDev& J, double x, double y, double z1) {
  const unsigned cx = (unsigned)__double2int_rd(st_dmul(x, J.inv_d));
  const unsigned cy = (unsigned)__double2int_rd(st_dmul(y, J.inv_d));
  const unsigned cz = (unsigned)__double2int_rd(st_dmul(z1, J.inv_d));
  return ((cx * 73856093u) ^ (cy * 19349663u) ^ (cz * 83492791u)) & (kCellHashBins - 1);
}

// Layered jobs (kWinLayers). z is not shifted by an oversample, so a deposit's lattice layer k_z is
// the same in all of them, and a sphere never leaves its layer: deposits ordered by layer can be cut
// into windows of whole layers that share no sphere, whatever the shift. Every sphere of such a
// window is complete when the window ends and is binned from shared memory, none goes through the
// spill log, and any range of windows is a work item of its own (a large job spreads over the CTAs
// without meeting in a table in HBM). The order is a counting sort: k_prep_count counts the z bins
// (lattice layers, or 2^k of them), k_prep_scan turns the counts into first places, and here each
// cell group of a block claims consecutive places in its bin, so that deposits of one cell stay
// together. The places a bin's groups get depend on the blocks' timing, the results do not (sums are
// exact). k_prep_pad cuts the windows.
// Measured against windows of the source order with boundary flags (per pass): 8 tracks of 4e6
// deposits, 10 nm, 50 oversamples 38.7 -> 25.4 ms; 16 of 1e6, 2 nm 27.1 -> 24.9; the
// single-precision mix 7.8 -> 7.0; one track of 300,007 deposits 327 -> 295 us. The uneven
// 2,048-track batch stays at 29.0 ms: its jobs of large spheres are not windowed.
//
// Four blocks per SM (64 registers, a few bytes of spills): the stage is memory-bound, and the
// fourth block's loads in flight are worth more than the spills cost.
__global__ void __launch_bounds__(kPrepThreads, 4) k_prep_write(PrepareParams p) {
  chain_start();
  const int64_t b = p.blk_base + blockIdx.x;
  const int j = prep_job(p, b);
  const JobDev J = p.jobs[j];
  const int64_t i0 = (b - p.blk_prefix[j]) * (int64_t)kPrepSlotsPerBlock;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kWarpsPerBlock = kPrepThreads / 32;
  constexpr int kRounds = kPrepSlotsPerBlock / kPrepThreads;
  constexpr int kGroupsPerThread = kPrepSlotsPerBlock / kPrepThreads;
  constexpr int kHashPerThread = kCellHashBins / kPrepThreads;
  __shared__ int s_warp[kRounds][kWarpsPerBlock];
  // sorted blocks: the first deposit (block-local index) of every cell-hash bin, and per group
  // (named by that first deposit) its size, then its offset
  __shared__ unsigned s_first[kCellHashBins];
  __shared__ unsigned s_group[kPrepSlotsPerBlock];
  __shared__ unsigned s_part[kWarpsPerBlock];
  // layered jobs: first place of each group, or with bit 31 its block bin and offset there
  __shared__ unsigned s_base[kPrepSlotsPerBlock];
  __shared__ int s_key[kBlockBins];          // block bins, the deposits of each and its first place
  __shared__ unsigned s_count[kBlockBins], s_place[kBlockBins];
  __shared__ unsigned short s_zbin[kPrepSlotsPerBlock];  // and its z bin
  int64_t run = p.blk_offset[b];  // kept index of the next kept deposit of this block
  const JobAux A = p.aux[j];
  const bool layered = A.windowed == kWinLayers;
  const bool sorted = p.sort == 2 || (p.sort == 1 && (J.flagged || layered));
  if (sorted) {
#pragma unroll
    for (int t = 0; t < kHashPerThread; ++t) s_first[threadIdx.x * kHashPerThread + t] = ~0u;
#pragma unroll
    for (int t = 0; t < kGroupsPerThread; ++t) s_group[threadIdx.x * kGroupsPerThread + t] = 0;
    if (threadIdx.x < kBlockBins) {
      s_key[threadIdx.x] = -1;
      s_count[threadIdx.x] = 0;
    }
  }
  const int E0 = choose_grid_exponent(A.e_min, A.e_max, J.n, A.flags & kAuxNonzero);
  unsigned created_cells = 0;  // cells this thread created (windowed jobs)
  // the loads of all rounds are issued before the block's one barrier, so each thread has all
  // of its source deposits in flight at once
  double x[kRounds], y[kRounds], z1[kRounds], e[kRounds];
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    const int64_t i = i0 + r * kPrepThreads + threadIdx.x;
    x[r] = 0; y[r] = 0; z1[r] = 0;
    if (i < J.n) {
      x[r] = J.x[i];
      y[r] = J.y[i];
      z1[r] = J.z[i];
    }
  }
  unsigned keep = 0, m[kRounds];
  unsigned slot_of[kRounds];  // sorted blocks: cell-hash bin, then group (high 16 bits) and rank
  if (sorted) __syncthreads();  // tables initialised
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    const int64_t i = i0 + r * kPrepThreads + threadIdx.x;
    z1[r] = st_dadd(z1[r], J.zsh);
    const bool k = i < J.n && fabs(z1[r]) < J.HL && fabs(x[r]) < J.xy_keep && fabs(y[r]) < J.xy_keep;
    keep |= k ? 1u << r : 0u;
    m[r] = __ballot_sync(0xffffffffu, k);
    if (lane == 0) s_warp[r][warp] = __popc(m[r]);
    e[r] = k ? J.edep[i] : 0.0;
    slot_of[r] = 0;
    if (sorted && k) {
      slot_of[r] = cell_hash_bin(J, x[r], y[r], z1[r]);
      atomicMin(&s_first[slot_of[r]], (unsigned)(r * kPrepThreads + threadIdx.x));
    }
  }
  __syncthreads();
  if (layered) {
    // Each group (named by its first deposit, which claims for it) takes consecutive places in
    // its z bin; a deposit whose hash collided with a group of another bin claims its own.
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
      const unsigned own = r * kPrepThreads + threadIdx.x;
      if (keep & (1u << r)) s_zbin[own] = (unsigned short)z_bin(J, z1[r]);
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
      if (keep & (1u << r)) {
        const unsigned own = r * kPrepThreads + threadIdx.x;
        const unsigned first = s_first[slot_of[r]];
        const unsigned g = s_zbin[first] == s_zbin[own] ? first : own;
        slot_of[r] = (g << 16) | atomicAdd(&s_group[g], 1u);
      }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
      const unsigned own = r * kPrepThreads + threadIdx.x;
      if ((keep & (1u << r)) && (slot_of[r] >> 16) == own) {
        const int bin = s_zbin[own], q = block_bin(s_key, bin);
        s_base[own] = q >= 0 ? 0x80000000u | q << 16 | atomicAdd(&s_count[q], s_group[own])
                             : atomicAdd(&p.bins[J.bin_off + bin], s_group[own]);
        ++created_cells;
      }
    }
    __syncthreads();
    if (threadIdx.x < kBlockBins && s_count[threadIdx.x])
      s_place[threadIdx.x] = atomicAdd(&p.bins[J.bin_off + s_key[threadIdx.x]], s_count[threadIdx.x]);
    __syncthreads();
  } else if (sorted) {
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
      if (keep & (1u << r)) {
        const unsigned g = s_first[slot_of[r]];
        slot_of[r] = (g << 16) | atomicAdd(&s_group[g], 1u);
      }
    }
    __syncthreads();
    // exclusive scan of the group sizes: each thread sums its kGroupsPerThread groups, the warps
    // scan the thread sums, and the warp totals are scanned in shared memory
    unsigned v[kGroupsPerThread], tsum = 0;
#pragma unroll
    for (int t = 0; t < kGroupsPerThread; ++t) {
      v[t] = s_group[threadIdx.x * kGroupsPerThread + t];
      tsum += v[t];
    }
    unsigned incl = tsum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned u = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += u;
    }
    if (lane == 31) s_part[warp] = incl;
    __syncthreads();
    unsigned base = incl - tsum;
    for (int w = 0; w < warp; ++w) base += s_part[w];
#pragma unroll
    for (int t = 0; t < kGroupsPerThread; ++t) {
      s_group[threadIdx.x * kGroupsPerThread + t] = base;
      base += v[t];
    }
    __syncthreads();
  }
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    int before = 0, total = 0;
#pragma unroll
    for (int w = 0; w < kWarpsPerBlock; ++w) {
      const int c = s_warp[r][w];
      before += (w < warp) ? c : 0;
      total += c;
    }
    uint64_t ckey = kEmptyKey;  // windowed jobs: the kept deposit's flag cell and window
    uint32_t cwin = 0;
    if (keep & (1u << r)) {
      // kept index: block order, or the position of the deposit's group and rank in sorted
      // blocks
      const unsigned first = layered ? s_base[slot_of[r] >> 16] : 0;
      const int64_t k = layered ? (int64_t)(first >> 31 ? s_place[first >> 16 & (kBlockBins - 1)] + (first & 0xFFFFu)
                                                        : first) + (slot_of[r] & 0xFFFFu)
                        : sorted ? p.blk_offset[b] + s_group[slot_of[r] >> 16] + (slot_of[r] & 0xFFFFu)
                               : run + before + __popc(m[r] & ((1u << lane) - 1u));
      const double az = st_dsub(z1[r], J.gSO);
      const double kd = lattice_index(az, J.d, J.inv_d);
      const double dz = st_dsub(st_dmul(kd, J.d), az);
      const int64_t dst = prep_slot(J, k);
      if (p.fp32) {
        reinterpret_cast<float2*>(p.PG)[dst] = make_float2(__double2float_rn(x[r]), __double2float_rn(y[r]));
        p.PGZ[dst] = __double2float_rn(st_dmul(dz, dz));
      } else {
        const double gz = st_dmul(dz, J.g_scale);
        p.PG[dst] = make_int2(__double2int_rn(st_dmul(x[r], J.g_scale)),
                              __double2int_rn(st_dmul(y[r], J.g_scale)));
        p.PGZ[dst] = __double2float_rn(st_dmul(gz, gz));
      }
      p.PSRC[dst] = (uint32_t)(i0 + r * kPrepThreads + threadIdx.x);
      uint64_t lo, hi;
      to_fixed(__ddiv_rn(e[r], J.denom), E0, &lo, &hi);
      p.PV[dst] = make_ulonglong2(lo, hi);
      p.PKEY[dst] = (uint64_t)(long long)kd * J.N2;
      if (A.windowed == kWinFlags) {
        ckey = cell_key(cell_of(x[r], y[r], z1[r], J.inv_cell), 0, 0, 0);
        cwin = (uint32_t)(k / kWindow);
      }
    }
    if (A.windowed == kWinFlags) {
      // adjacent lanes hold adjacent source deposits, which on dense tracks share a cell and a
      // window: an insert equal to the previous lane's changes nothing and is skipped, which
      // spares the cell's slot most of its same-address atomics
      const uint64_t pkey = __shfl_up_sync(0xffffffffu, ckey, 1);
      const uint32_t pwin = __shfl_up_sync(0xffffffffu, cwin, 1);
      if (ckey != kEmptyKey && !(lane > 0 && pkey == ckey && pwin == cwin))
        created_cells += cell_insert(p, J, ckey, cwin);
    }
    run += total;
  }
  if (A.windowed) {  // occupied cells, one addition per block (the window size depends on them)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) created_cells += __shfl_xor_sync(0xffffffffu, created_cells, o);
    __shared__ unsigned s_cells;
    if (threadIdx.x == 0) s_cells = 0;
    __syncthreads();
    if (lane == 0 && created_cells) atomicAdd(&s_cells, created_cells);
    __syncthreads();
    if (threadIdx.x == 0 && s_cells) atomicAdd(&p.aux[j].cells, (unsigned long long)s_cells);
  }
}

// One block per job: padding slots [kept, kept rounded up to a warp tile), and the window list of
// a layered job.
__global__ void __launch_bounds__(kWarpTile) k_prep_pad(PrepareParams p) {
  chain_start();
  const int j = blockIdx.x;
  const JobDev J = p.jobs[j];
  const long long kept = p.aux[j].kept;
  if (p.aux[j].windowed == kWinLayers) {
    __shared__ uint32_t s_ends[kMaxBins];
    for (int b = threadIdx.x; b < J.n_bins; b += kWarpTile) s_ends[b] = p.bins[J.bin_off + b];
    __syncthreads();
    if (threadIdx.x < 32) cut_windows(p, J, &p.aux[j], s_ends);
  }
  if ((kept % kWarpTile) == 0) return;
  const long long k = kept + threadIdx.x;
  if (k >= (kept / kWarpTile + 1) * kWarpTile) return;
  const int64_t dst = prep_slot(J, k);
  if (p.fp32) {
    reinterpret_cast<float2*>(p.PG)[dst] = make_float2(__int_as_float(0x7FC00000), __int_as_float(0x7FC00000));
  } else {
    p.PG[dst] = make_int2(INT_MIN, INT_MIN);  // outside the voxel for every shift, without FP64
  }
  p.PGZ[dst] = __int_as_float(0x7F800000);
  p.PV[dst] = make_ulonglong2(0, 0);
  p.PKEY[dst] = 0;
}

// Boundary flags of the kept deposits of flagged jobs: a deposit is a boundary deposit when one of
// the flag cells around it (27 of side d, or eight of side 2d chosen by cell_nbr) holds a
// deposit of another window. A sphere whose hits in a window are
// all non-boundary has no hit in any other window (its hits are within distance d of each other),
// so the fused kernel can bin it as soon as the window is done.
// Eight blocks per SM (32 registers): the cell probes are L2 latency, which more warps hide.
__global__ void __launch_bounds__(kPrepThreads, 8) k_prep_flag(PrepareParams p) {
  chain_start();
  if (!*p.any_flags) return;
  const int64_t b = p.blk_base + blockIdx.x;
  const int j = prep_job(p, b);
  const JobDev J = p.jobs[j];
  const JobAux A = p.aux[j];
  if (A.windowed != kWinFlags) return;
  const int shift = coarse_windows(J, A) ? 1 : 0;
  const int64_t k0 = p.blk_offset[b];
  const int cnt = p.blk_count[b];
  for (int q = threadIdx.x; q < cnt; q += kPrepThreads) {
    const int64_t k = k0 + q;
    const int64_t dst = prep_slot(J, k);
    const uint32_t src = p.PSRC[dst];
    const double x = J.x[src], y = J.y[src], z = st_dadd(J.z[src], J.zsh);
    const uint32_t win = (uint32_t)(k / kWindow);
    bool boundary = false;
    // batches unrolled, so that the neighbour offsets are constants
    if (J.cell_nbr8) {
      const NbrOffsets o = nbr_offsets8(cell_nbr(x, y, z, J.inv_cell));
      const auto key_of = [&](int c) { return nbr_key8(o, c); };
#pragma unroll
      for (int c0 = 0; c0 < 8; c0 += 2)
        if (!boundary) boundary = cells_foreign<2>(p, J, key_of, c0, win, shift);
    } else {
      const uint64_t base = cell_key(cell_of(x, y, z, J.inv_cell), 0, 0, 0);
      const auto key_of = [&](int c) { return nbr_key27(base, c); };
#pragma unroll
      for (int c0 = 0; c0 < 27; c0 += 3)
        if (!boundary) boundary = cells_foreign<3>(p, J, key_of, c0, win, shift);
    }
    if (boundary) p.PKEY[dst] |= kBoundaryBit;
  }
}

// ---------------------------------------------------------------------------------------------
// Exact 128-bit accumulators
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void acc_add(unsigned long long* lo_p, unsigned long long* hi_p,
                                        uint64_t lo, uint64_t hi) {
  const unsigned long long old = atomicAdd(lo_p, (unsigned long long)lo);
  const unsigned long long h = hi + ((old + lo < old) ? 1ull : 0ull);
  if (h) atomicAdd(hi_p, h);
}

// The same on a shared-memory accumulator, whose low 64 bits are the words *w0 and *w1: a chain of
// 32-bit additions, each passing its carry on (unsigned wrap-around of the returned old value).
// Shared memory adds 32-bit words natively; a 64-bit addition is a compare-and-swap loop, which one
// SM ran at 18 clocks per warp on random slots and 188 on 16 contended ones, against 5.6 and 7.6 for
// two chained words. The high words only take a carry or a contribution beyond 64 bits.
// Uneven 2,048-track batch, fused kernel: 28.6 -> 26.5 ms; dense 2 nm ions 25.7 -> 25.4 ms.
__device__ __forceinline__ void smem_acc_add(unsigned int* w0, unsigned int* w1,
                                             unsigned long long* hi_p, uint64_t lo, uint64_t hi) {
  const unsigned int a0 = (unsigned int)lo;
  const unsigned int o0 = atomicAdd(w0, a0);
  const uint64_t s1 = (lo >> 32) + (o0 + a0 < o0 ? 1u : 0u);
  const unsigned int o1 = atomicAdd(w1, (unsigned int)s1);
  const uint64_t h = hi + (s1 >> 32) + (((uint64_t)o1 + (unsigned int)s1) >> 32);
  if (h) {
    unsigned int* w2 = reinterpret_cast<unsigned int*>(hi_p);
    const unsigned int a2 = (unsigned int)h;
    const unsigned int o2 = atomicAdd(w2, a2);
    const unsigned int a3 = (unsigned int)(h >> 32) + (o2 + a2 < o2 ? 1u : 0u);
    if (a3) atomicAdd(w2 + 1, a3);
  }
}

__device__ __forceinline__ void add128(uint64_t& alo, uint64_t& ahi, uint64_t lo, uint64_t hi) {
  const uint64_t s = alo + lo;
  ahi += hi + (s < alo ? 1ull : 0ull);
  alo = s;
}

// Spill-table insert (HBM). Returns false when the table has no free slot.
__device__ __forceinline__ bool gtable_add(uint64_t* gk, unsigned long long* glo,
                                           unsigned long long* ghi, uint32_t* gused,
                                           unsigned int* gcnt, uint32_t gcap, uint64_t key,
                                           uint64_t lo, uint64_t hi) {
  const uint32_t mask = gcap - 1;
  uint32_t h = slot_hash(key, mask);
  for (uint32_t probe = 0; probe < gcap; ++probe) {
    const uint64_t k = __ldcg((const unsigned long long*)&gk[h]);
    if (k == key) { acc_add(&glo[h], &ghi[h], lo, hi); return true; }
    if (k == kEmptyKey) {
      const uint64_t old = atomicCAS((unsigned long long*)&gk[h], kEmptyKey, key);
      if (old == kEmptyKey) {
        const unsigned idx = atomicAdd(gcnt, 1u);
        gused[idx] = h;
        acc_add(&glo[h], &ghi[h], lo, hi);
        return true;
      }
      if (old == key) { acc_add(&glo[h], &ghi[h], lo, hi); return true; }
    }
    h = (h + 1) & mask;
  }
  return false;
}

// Four consecutive 8-byte records (32 bytes, 32-byte aligned: a lane's deposits of a tile) with one
// 256-bit read-only load. (k_fused reads all its records through the non-coherent path, so it is never
// launched chained: they have to stay as they are from its start on. Plain loads, which would allow
// it, cost the 2,048-track batch 27.2 -> 29.7 ms; the link they would save is about 1 us.)
__device__ __forceinline__ void ldg_records(const int2* p, unsigned long long* v) {
  asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];"
      : "=l"(v[0]), "=l"(v[1]), "=l"(v[2]), "=l"(v[3])
      : "l"(p));
}

// Dynamic shared memory of the fused kernel. The sphere table sits at fixed offsets (so that its
// addresses cost no registers): keys, low and high accumulator words, the used-slot list and the
// boundary bitmap; the shared-memory histogram (y*f(y), edges, counts) follows it.
extern __shared__ __align__(16) unsigned char smem_raw[];

template <int CAP>
struct SmemTable {
  __device__ __forceinline__ static uint64_t* keys() { return reinterpret_cast<uint64_t*>(smem_raw); }
  // low 64 bits of a slot's sum, as two arrays of 32-bit words
  __device__ __forceinline__ static unsigned int* lo0() {
    return reinterpret_cast<unsigned int*>(smem_raw + 8 * CAP);
  }
  __device__ __forceinline__ static unsigned int* lo1() {
    return reinterpret_cast<unsigned int*>(smem_raw + 12 * CAP);
  }
  __device__ __forceinline__ static uint64_t lo(uint32_t h) {
    return ((uint64_t)lo1()[h] << 32) | lo0()[h];
  }
  __device__ __forceinline__ static unsigned long long* hi() {
    return reinterpret_cast<unsigned long long*>(smem_raw + 16 * CAP);
  }
  __device__ __forceinline__ static uint16_t* used() {
    return reinterpret_cast<uint16_t*>(smem_raw + 24 * CAP);
  }
  // CAP bits: the entry holds a boundary deposit's contribution
  __device__ __forceinline__ static unsigned int* flags() {
    return reinterpret_cast<unsigned int*>(smem_raw + 26 * CAP);
  }
  __device__ __forceinline__ static double* hist() {
    return reinterpret_cast<double*>(smem_raw + 26 * CAP + CAP / 8);
  }
  __device__ __forceinline__ static void clear(uint32_t h) {
    keys()[h] = kEmptyKey;
    lo0()[h] = 0;
    lo1()[h] = 0;
    hi()[h] = 0;
  }
};

// Occupancy and overflow of the sphere table are counted per window in one of three rotating
// slots (window i uses slot i % 3; a job without window flags always uses slot 0): the slot of the
// next window can then be cleared while the current window's is still being read, which saves a
// CTA barrier per window.
struct CtaState {
  int item;
  int tc[3];        // used slots of the table (the used-list length) in this window
  int spilled;      // some sphere of this oversample has a partial sum in the spill table
  int ovf[3];       // this window sent a contribution to the spill table directly
  int edges_hist;   // histogram whose edges are in shared memory (-1: none)
  int log_mode;     // private item: table overflows, flushes and window-end spills go to the log
  int logn;         // records in the spill log of this oversample
  int table;        // spill table that the CTA holds for its private items (-1: none)
  long long hist_work;  // deposit*oversamples in the shared-memory histogram
  int hist_span;      // its sum_span
  double sx, sy;      // shift of the current oversample, and in lattice units plus half a cell
  int cx, cy;
};

// Spill table of the current item: the CTA's table restricted to a power-of-two prefix sized
// for the item's job, so that small jobs touch a small, cache-friendly region.
struct Spill {
  uint64_t* keys;
  unsigned long long* lo;
  unsigned long long* hi;
  uint32_t* used;
  unsigned int* count;
  uint32_t cap;
};

// Appends a sphere's partial sum to the CTA's spill log: the first half of the item's spill table
// holds (key, lo, hi) records in arrival order, written with plain stores, so a window end does
// not wait for global atomics. A log takes at most one record per hit of its oversample, and the
// table has at least two slots per kept deposit, so it cannot run out.
__device__ __forceinline__ void log_append(CtaState* cs, const FusedParams& P, const Spill& G,
                                           uint64_t key, uint64_t lo, uint64_t hi) {
  const unsigned idx = (unsigned)atomicAdd(&cs->logn, 1);
  if (idx < G.cap / 2) {
    G.keys[idx] = key;
    G.lo[idx] = lo;
    G.hi[idx] = hi;
  } else {
    atomicOr(P.error_flags, 1);
  }
}

// Adds a contribution to the CTA's shared-memory table. A sphere already in the table is always
// found there; a new one is refused (false) when the table is three quarters full or its probe
// sequence is too long.
template <int CAP>
__device__ __forceinline__ bool table_insert(const SmemTable<CAP>& T, CtaState* cs, uint64_t key,
                                             uint64_t lo, uint64_t hi, bool boundary, int slot) {
  constexpr int kHardLimit = (CAP * 3) / 4;
  uint32_t h = table_hash(key, CAP - 1);
#pragma unroll 1
  for (int probe = 0; probe < 32; ++probe) {
    const uint64_t k = ((volatile uint64_t*)T.keys())[h];
    bool mine = k == key;
    if (!mine && k == kEmptyKey) {
      if (*(volatile int*)&cs->tc[slot] >= kHardLimit) return false;
      const uint64_t old = atomicCAS((unsigned long long*)&T.keys()[h], kEmptyKey, key);
      if (old == kEmptyKey) {
        const int idx = atomicAdd(&cs->tc[slot], 1);
        T.used()[idx] = (uint16_t)h;
      }
      mine = old == kEmptyKey || old == key;
    }
    if (mine) {
      smem_acc_add(&T.lo0()[h], &T.lo1()[h], &T.hi()[h], lo, hi);
      if (boundary) atomicOr(&T.flags()[h >> 5], 1u << (h & 31));
      return true;
    }
    h = (h + 1) & (CAP - 1);
  }
  return false;
}

// Adds one sphere contribution to the shared-memory table, or, when the table refuses it, to the
// spill log (window-flagged private items) or the spill table. Jobs with window flags empty the
// table at every window end; other jobs keep their spheres for the whole oversample, and on the
// 4096-slot table are also flushed at window ends once it is half full (window_checks).
template <int CAP>
__device__ __forceinline__ void sphere_add(const SmemTable<CAP>& T, CtaState* cs,
                                           const FusedParams& P, const Spill& G, uint64_t key,
                                           uint64_t lo, uint64_t hi, bool boundary, int slot) {
  if (table_insert<CAP>(T, cs, key, lo, hi, boundary, slot)) return;
  *(volatile int*)&cs->ovf[slot] = 1;
  if (*(volatile int*)&cs->log_mode) {
    log_append(cs, P, G, key, lo, hi);
    return;
  }
  *(volatile int*)&cs->spilled = 1;
  if (!gtable_add(G.keys, G.lo, G.hi, G.used, G.count, G.cap, key, lo, hi))
    atomicOr(P.error_flags, 1);
}

constexpr int kHistCopies = 4;   // at most this many shared-memory copies of a histogram

struct BinContext {
  const double* edges;    // shared-memory copy when the histogram fits, else HBM
  unsigned long long* gcounts;
  double* gyfy;
  unsigned int* hcount;   // null: accumulate straight into HBM
  unsigned long long* hylo;  // y*f(y) per bin: 128-bit sum on the bin's grid (see bin_sphere)
  unsigned long long* hyhi;
  int copies;             // shared-memory copies of the histogram, used by warp % copies
  int nbins;
  int mode;               // 0: linear candidate, 1: log2 candidate
  double ca, cb;          // candidate bin = (y - ca) * cb, or (log2 y - ca) * cb
  int E0;
  int job;
  int span;               // sum_span of the shared-memory histogram
  double scale;           // 2^E0, or 0 when E0 is near the ends of the exponent range
};

// HistogramRange bin of y (edges[b] <= y < edges[b+1], else -1) from a guess b that was off.
__device__ __forceinline__ int find_bin_near(const double* e, int nb, int b, double y) {
  if (!(y >= e[0]) || !(y < e[nb])) return -1;
#pragma unroll 1
  for (int it = 0; it < 8; ++it) {
    if (y < e[b]) { --b; continue; }
    if (y >= e[b + 1]) { ++b; continue; }
    return b;
  }
  int l = 0, h = nb;  // far-off guess: binary search
  while (h - l > 1) {
    const int m = (l + h) >> 1;
    if (e[m] <= y) l = m; else h = m;
  }
  return l;
}

// What binning a sphere reads of its context, in registers: the shared-memory adds of the loop that
// bins a window's spheres would make the compiler read the context again for every sphere. With the
// short cuts below for sums under 2^64 and for y near its bin's edge (both exact), fused time of the
// uneven 2,048-track batch 24.9 -> 23.7 ms, of 16 tracks of 1e6 deposits, 2 nm 23.2 -> 21.6.
struct BinRegs {
  const double* edges;
  double scale;
  float ca, cb;   // bin guess (a float suffices: the edges decide)
  int nbins, mode;
  int copy;       // first bin of this warp's copy of the histogram, -1: straight into HBM

  __device__ __forceinline__ explicit BinRegs(const BinContext& B)
      : edges(B.edges), scale(B.scale), ca((float)B.ca), cb((float)B.cb), nbins(B.nbins),
        mode(B.mode) {
    // warps spread over the copies, so that fewer of them contend for a bin
    copy = B.hcount ? (int)((threadIdx.x >> 5) % (unsigned)B.copies) * nbins : -1;
  }
};

template <typename KeyOf>
__device__ __forceinline__ void bin_sphere(const BinRegs& R, const BinContext& B,
                                           const FusedParams& P, const KeyOf& key_of,
                                           uint64_t lo, uint64_t hi, unsigned int& spheres,
                                           unsigned int& binned, int os) {
  // (double)lo * 2^E0 is exact after the one rounding when the sum is below 2^64 and 2^E0 is far
  // from the exponent range's ends
  const double y = hi == 0 && R.scale != 0.0 ? st_dmul(u64_to_double_rn(lo), R.scale)
                                             : from_fixed(lo, hi, B.E0);
  ++spheres;
  const float yf = (float)y;
  const float t = ((R.mode ? __log2f(yf) : yf) - R.ca) * R.cb;
  int b = t >= 0.f ? (t < (float)R.nbins ? (int)t : R.nbins - 1) : 0;
  double e0 = R.edges[b];
  if (!(y >= e0) || !(y < R.edges[b + 1])) {
    b = find_bin_near(R.edges, R.nbins, b, y);
    e0 = b >= 0 ? R.edges[b] : 0.0;
  }
  if (b >= 0) {
    ++binned;
    if (R.copy >= 0) {
      const int c = R.copy + b;
      atomicAdd(&B.hcount[c], 1u);
      // y >= edge_b > 0 is a whole multiple of ulp(edge_b): its sum is kept exactly as a 128-bit
      // integer on that grid, with integer atomics (a double atomic add is a retry loop under
      // contention). A bin whose lower edge is not a positive normal number keeps a double sum
      // in the low word instead.
      const uint64_t eb = (uint64_t)__double_as_longlong(e0);
      if ((int64_t)eb > 0 && (eb >> 52) != 0) {
        uint64_t lo = 0, hi = 0;
        const uint64_t yb = (uint64_t)__double_as_longlong(y);
        const int up = (int)(yb >> 52) - (int)(eb >> 52);  // y >= edge_b: not negative
        if (up < 12) lo = ((yb & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull) << up;
        else if (up <= B.span) to_fixed(y, (int)(eb >> 52) - 1075, &lo, &hi);
        else atomicAdd(&B.gyfy[b], y);  // the copy's 128 bits could not hold the sum
        unsigned int* w = reinterpret_cast<unsigned int*>(&B.hylo[c]);
        smem_acc_add(w, w + 1, &B.hyhi[c], lo, hi);
      } else {
        atomicAdd(reinterpret_cast<double*>(&B.hylo[c]), y);
      }
    } else {
      atomicAdd(&B.gcounts[b], 1ull);
      atomicAdd(&B.gyfy[b], y);
    }
  }
  if (P.export_buf) {
    const unsigned long long idx = atomicAdd(P.export_count, 1ull);
    if (idx < P.export_cap) {
      SphereRecord r;
      r.key = key_of();
      r.y = y;
      r.os = os;
      r.job = B.job;
      P.export_buf[idx] = r;
    } else {
      atomicOr(P.error_flags, 2);
    }
  }
}

// Appends every shared-memory entry to the spill log and empties the shared table.
template <int CAP, int THREADS>
__device__ __forceinline__ void flush_to_log(const SmemTable<CAP>& T, int cnt, CtaState* cs,
                                             const FusedParams& P, const Spill& G) {
  for (int i = threadIdx.x; i < cnt; i += THREADS) {
    const uint32_t h = T.used()[i];
    log_append(cs, P, G, T.keys()[h], T.lo(h), T.hi()[h]);
    T.clear(h);
  }
}

// Moves every shared-memory entry into the spill table and empties the shared table.
template <int CAP, int THREADS>
__device__ __forceinline__ void flush_to_spill(const SmemTable<CAP>& T, int cnt,
                                               const FusedParams& P, const Spill& G) {
  for (int i = threadIdx.x; i < cnt; i += THREADS) {
    const uint32_t h = T.used()[i];
    if (!gtable_add(G.keys, G.lo, G.hi, G.used, G.count, G.cap, T.keys()[h], T.lo(h), T.hi()[h]))
      atomicOr(P.error_flags, 1);
    T.clear(h);
  }
}

// ---------------------------------------------------------------------------------------------
// Spill-table pool: one table per CTA of the launch. A CTA holds at most one table at a time
// (for its private item, or for the shared unit it works on until the unit is binned), so a free
// table always exists; the bounded scan only guards against a logic error.
// ---------------------------------------------------------------------------------------------
__device__ int pool_acquire(unsigned int* bits, int n_tables, int* err) {
  const int words = (n_tables + 31) / 32;
  for (int attempt = 0; attempt < 64; ++attempt) {
    for (int w = 0; w < words; ++w) {
      const unsigned valid = (w == words - 1 && (n_tables & 31)) ? ((1u << (n_tables & 31)) - 1u) : ~0u;
      unsigned freeb = ~__ldcg(&bits[w]) & valid;
      while (freeb) {
        const int b = __ffs(freeb) - 1;
        const unsigned old = atomicOr(&bits[w], 1u << b);
        if (!(old & (1u << b))) return w * 32 + b;
        freeb &= ~(1u << b);
      }
    }
  }
  atomicOr(err, 4);
  return -1;
}

__device__ __forceinline__ void pool_release(unsigned int* bits, int t) {
  atomicAnd(&bits[t >> 5], ~(1u << (t & 31)));
}

// Table of shared unit u: the first helper acquires it, the others wait (bounded: max_polls
// sleeps of at least 64 ns) until it is published. A wait that runs out sets error flag 8 and
// returns -1, and the item is given up; the host reports the run as ST_ERR_DEVICE_WAIT.
constexpr long long kUnitWaitPolls = 1ll << 24;
__device__ int unit_table_get(const FusedParams& P, int u, long long max_polls = kUnitWaitPolls) {
  int t = atomicCAS(&P.unit_table[u], -1, -2);
  if (t == -1) {
    t = pool_acquire(P.pool_bits, gridDim.x, P.error_flags);
    atomicExch(&P.unit_table[u], t < 0 ? -3 : t);
    return t;
  }
  for (long long spin = 0; t == -2 && spin < max_polls; ++spin) {
    __nanosleep(64);
    t = *(volatile int*)&P.unit_table[u];
  }
  if (t < 0) { atomicOr(P.error_flags, 8); return -1; }
  return t;
}

__device__ __forceinline__ Spill spill_of(const FusedParams& P, int t, long long kept) {
  Spill G;
  G.keys = P.gkeys + (size_t)t * P.gcap;
  G.lo = P.glo + (size_t)t * P.gcap;
  G.hi = P.ghi + (size_t)t * P.gcap;
  G.used = P.gused + (size_t)t * P.gcap;
  G.count = P.gcount + t;
  uint32_t cap = 1024;
  while (cap < P.gcap && (long long)cap < 2 * kept) cap <<= 1;
  G.cap = cap;
  return G;
}

// Bins and clears every entry of a spill table (all threads of the CTA).
template <int THREADS>
__device__ __forceinline__ void bin_spill(const Spill& G, const BinContext& B, const FusedParams& P,
                                          unsigned int& spheres, unsigned int& binned, int os) {
  const unsigned gc = __ldcg(G.count);
  const BinRegs BR(B);
  for (unsigned i = threadIdx.x; i < gc; i += THREADS) {
    const uint32_t h = __ldcg(&G.used[i]);
    const uint64_t key = __ldcg((const unsigned long long*)&G.keys[h]);
    const uint64_t lo = __ldcg(&G.lo[h]);
    const uint64_t hi = __ldcg(&G.hi[h]);
    bin_sphere(BR, B, P, [&] { return key; }, lo, hi, spheres, binned, os);
    G.keys[h] = kEmptyKey; G.lo[h] = 0; G.hi[h] = 0;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    *G.count = 0;
    __threadfence();
  }
}

// Partition of a spill-log record: a hash of the key independent of the table's slot hash.
__device__ __forceinline__ int log_part(uint64_t key, int parts) {
  return (int)(((uint64_t)(uint32_t)((key * 0xD6E8FEB86659FD93ull) >> 32) * (uint64_t)parts) >> 32);
}

// One reduction pass: the records [r0, r1) of R whose partition is `part` (all of them when
// parts is 1) are summed in the empty shared table and binned. If the table refused any record,
// the pass's spheres go whole to the hash table F instead (binned last), so that no sphere is
// split between the two. Returns whether F received anything (the same in every thread).
template <int CAP, int THREADS>
__device__ __forceinline__ int log_pass(const SmemTable<CAP>& T, CtaState& cs,
                                        const FusedParams& P, const Spill& R, int r0, int r1,
                                        int part, int parts, const Spill& F, int slot,
                                        const BinContext& B, unsigned int& spheres,
                                        unsigned int& binned, int os) {
  const int tid = threadIdx.x;
  int refused = 0;
  // four records in flight per thread before any is inserted
  for (int i0 = r0 + tid; i0 < r1; i0 += 4 * THREADS) {
    uint64_t kk[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + u * THREADS;
      kk[u] = i < r1 ? __ldcg((const unsigned long long*)&R.keys[i]) : kEmptyKey;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + u * THREADS;
      if (i >= r1 || (parts > 1 && log_part(kk[u], parts) != part)) continue;
      const uint64_t lo = __ldcg(&R.lo[i]), hi = __ldcg(&R.hi[i]);
      if (!table_insert<CAP>(T, &cs, kk[u], lo, hi, false, slot)) {
        if (!gtable_add(F.keys, F.lo, F.hi, F.used, F.count, F.cap, kk[u], lo, hi))
          atomicOr(P.error_flags, 1);
        refused = 1;
      }
    }
  }
  refused = __syncthreads_or(refused);
  const int cnt = cs.tc[slot];
  if (tid == 0) cs.tc[(slot + 1) % 3] = 0;  // the next pass's slot: last read two passes ago
  const BinRegs BR(B);
  for (int i = tid; i < cnt; i += THREADS) {
    const uint32_t h = T.used()[i];
    if (refused) {
      if (!gtable_add(F.keys, F.lo, F.hi, F.used, F.count, F.cap, T.keys()[h], T.lo(h), T.hi()[h]))
        atomicOr(P.error_flags, 1);
    } else {
      bin_sphere(BR, B, P, [&] { return T.keys()[h]; }, T.lo(h), T.hi()[h], spheres, binned, os);
    }
    T.clear(h);
  }
  __syncthreads();
  return refused;
}

// End of a window-flagged private oversample: sums the spill log (the first half of the spill
// table, records [0, L)) per sphere and bins it, in passes of at most CAP / 2 records (a pass has
// no more distinct keys than records, so the table stays at most half full).
//  - Bucketed (more than one pass, and the per-pass counts fit the table's used-slot list, free at
//    this point): the records are counted per hash partition, scattered into buckets in the second
//    half of the spill table, and each bucket is summed in one pass; the emptied first half is the
//    fallback table, and the bucket bounds sit in the spill table's used list beyond its reach.
//  - Otherwise every pass scans the whole log for its partition, with the second half of the
//    spill table as the fallback.
// Every record is cleared again for the pool's next user.
template <int CAP, int THREADS>
__device__ __forceinline__ void log_reduce(const SmemTable<CAP>& T, CtaState& cs,
                                           const FusedParams& P, const Spill& G,
                                           const BinContext& B, unsigned int& spheres,
                                           unsigned int& binned, int os) {
  const int tid = threadIdx.x;
  const int L = cs.logn;  // read after superimpose's closing barrier: the same in every thread
  if (L == 0) return;
  constexpr int kPart = CAP / 2;  // records per pass
  const int parts = (L + kPart - 1) / kPart;
  Spill lo_half = G, hi_half = G;
  lo_half.cap = G.cap / 2;
  hi_half.keys += G.cap / 2;
  hi_half.lo += G.cap / 2;
  hi_half.hi += G.cap / 2;
  hi_half.cap = G.cap / 2;
  if (tid == 0) for (int k = 0; k < 3; ++k) cs.tc[k] = 0;
  __syncthreads();
  int any_out = 0;
  if (parts == 1 || 2 * parts > CAP / 2) {
    for (int q = 0; q < parts; ++q)
      any_out |= log_pass<CAP, THREADS>(T, cs, P, lo_half, 0, L, q, parts, hi_half, q % 3, B,
                                        spheres, binned, os);
    for (int i = tid; i < L; i += THREADS) { G.keys[i] = kEmptyKey; G.lo[i] = 0; G.hi[i] = 0; }
    if (any_out) bin_spill<THREADS>(hi_half, B, P, spheres, binned, os);
  } else {
    unsigned int* cnt = reinterpret_cast<unsigned int*>(T.used());  // parts counts, parts cursors
    uint32_t* bounds = G.used + G.cap / 2;                              // parts + 1 bucket bounds
    for (int i = tid; i < 2 * parts; i += THREADS) cnt[i] = 0;
    __syncthreads();
    for (int i = tid; i < L; i += THREADS)
      atomicAdd(&cnt[log_part(__ldcg((const unsigned long long*)&G.keys[i]), parts)], 1u);
    __syncthreads();
    if (tid == 0) {
      unsigned run = 0;
      for (int q = 0; q < parts; ++q) {
        bounds[q] = run;
        cnt[parts + q] = run;
        run += cnt[q];
      }
      bounds[parts] = run;
    }
    __syncthreads();
    for (int i = tid; i < L; i += THREADS) {
      const uint64_t key = __ldcg((const unsigned long long*)&G.keys[i]);
      const uint64_t lo = __ldcg(&G.lo[i]), hi = __ldcg(&G.hi[i]);
      const unsigned pos = atomicAdd(&cnt[parts + log_part(key, parts)], 1u);
      hi_half.keys[pos] = key; hi_half.lo[pos] = lo; hi_half.hi[pos] = hi;
      G.keys[i] = kEmptyKey; G.lo[i] = 0; G.hi[i] = 0;
    }
    __syncthreads();  // buckets written, the first half empty again (the fallback from here on)
    for (int q = 0; q < parts; ++q) {
      const int r0 = (int)__ldcg(&bounds[q]), r1 = (int)__ldcg(&bounds[q + 1]);
      any_out |= log_pass<CAP, THREADS>(T, cs, P, hi_half, r0, r1, q, 1, lo_half, q % 3, B,
                                        spheres, binned, os);
    }
    for (int i = tid; i < L; i += THREADS) {
      hi_half.keys[i] = kEmptyKey; hi_half.lo[i] = 0; hi_half.hi[i] = 0;
    }
    if (any_out) bin_spill<THREADS>(lo_half, B, P, spheres, binned, os);
  }
  __syncthreads();
  if (tid == 0) {
    for (int k = 0; k < 3; ++k) cs.tc[k] = 0;
    cs.logn = 0;
  }
  __syncthreads();
}

struct FusedJob {
  JobDev J;
  int windowed;     // kWinNone, kWinFlags or kWinLayers
  const unsigned long long* wins;  // layered jobs: the window list, else null
  int win_tiles;    // warp tiles per warp in a window: kWinTiles, or kCoarseTiles
};

// Superimposes oversample `os` of a job over warp tiles [wt_begin, wt_end) (whole windows):
// shift, box test, lattice test, key, exact run / shared-memory reduction. For layered jobs the
// range is one of windows of F.wins instead. For windowed jobs every window ends by binning its
// complete spheres and moving boundary spheres to G (layered jobs have none, except the parts of a
// bin larger than a window whose spheres fill the table); otherwise
// spheres accumulate across windows and the shared table spills to G when it fills up.
// F32: the FP32 geometry variant (x, y, shifts, lattice index and distance in float; z part of
// the distance, keys and energies as in the FP64 form).
template <int CAP, int THREADS, bool F32>
__device__ __forceinline__ void superimpose(const FusedParams& P, const FusedJob& F,
                                            const SmemTable<CAP>& T, CtaState& cs,
                                            const Spill& G, const BinContext& B, int os,
                                            int64_t begin, int64_t end,
                                            unsigned int& hits, unsigned int& inbox,
                                            unsigned int& spheres, unsigned int& binned) {
  constexpr int kWarps = THREADS / 32;
  const JobDev& J = F.J;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool windowed = F.windowed != kWinNone;
  const unsigned long long* const wins = F.wins;
  const int64_t base = J.prep_off + 4 * lane;
  const uint32_t N = J.N;
  // F32: x' = x + sx, box |x'| < HL', a = x' - gSO, k = rint(a * (1/d)), dx = k*d - a,
  // hit iff (dx^2 + dy^2) + dz^2 <= r^2, every step rounded to float
  const float sxf = __double2float_rn(cs.sx), syf = __double2float_rn(cs.sy);
  const float fHL = J.f_HL, fgSO = J.f_gSO, fd = J.f_d, finv = J.f_inv_d, fr2 = J.f_r2;
  // FP64 form: integer geometry (set_integer_geometry). An offset below 2^22 becomes a float by
  // its bits under the exponent of 2^23, less 2^23 and half a cell.
  const int S = F32 ? 0 : J.g_shift;
  const int cx = cs.cx, cy = cs.cy;
  const unsigned in_max = (unsigned)J.g_ns - 4u, near_max = (unsigned)J.g_ns + 2u;
  const unsigned low = (1u << S) - 1u;
  const float centre = 8388608.0f + (float)(1 << S) * 0.5f;
  const float lo2 = J.g_lo, hi2 = J.g_hi;

  // Jobs without window flags on the 8192-slot table run their windows without a barrier (a CTA
  // barrier per window cost more than the occasional new sphere sent to the spill table by a
  // full table); on the 4096-slot table, a job whose whole lattice (N^3 spheres) exceeds the flush
  // threshold checks the table at every window end and flushes it to the spill table
  const bool log_mode = cs.log_mode != 0;
  const bool window_checks = CAP < 2 * kCtaTile && !windowed &&
                             (uint64_t)J.N * J.N2 > (uint64_t)P.flush_threshold;
  int wi = 0;  // emptied windows within this call
  bool logged = false;  // part of the current layer bin is in the spill log
  for (int64_t at = begin; at < end;) {
    const int slot = windowed ? wi % 3 : 0;
    // the window's warp tiles [w0, w1): win_tiles per warp from tile `at`, or window `at` of the
    // list, which may begin and end inside a tile (clip0: its first deposit in tile w0, clip1:
    // one past its last in tile w1 - 1)
    int w0, w1, clip0 = 0, clip1 = kWarpTile;
    bool more = false;  // the next window continues this one's last bin
    if (wins) {
      const unsigned long long a = __ldg(&wins[at]), b = __ldg(&wins[at + 1]);
      const long long k0 = (long long)(a & ~kWinContinues), k1 = (long long)(b & ~kWinContinues);
      more = (b & kWinContinues) != 0;
      w0 = (int)(k0 / kWarpTile);
      w1 = (int)((k1 + kWarpTile - 1) / kWarpTile);
      clip0 = (int)(k0 % kWarpTile);
      clip1 = (int)(k1 - (long long)(w1 - 1) * kWarpTile);
      ++at;
    } else {
      w0 = (int)at;
      at = at + kWarps * F.win_tiles < end ? at + kWarps * F.win_tiles : end;
      w1 = (int)at;
    }
#pragma unroll 1
    for (int w = w0 + warp; w < w1; w += kWarps) {
      {
        const int64_t tb = base + (int64_t)w * kWarpTile;  // this lane's deposits: tb .. tb + 3
        int kxv[kDepPerLane], kyv[kDepPerLane];            // lattice indices, shifted by S
        unsigned hitmask = 0, boxmask = 0;
        unsigned long long g[kDepPerLane];
        ldg_records(P.PG + tb, g);
        const float4 gz = __ldg(reinterpret_cast<const float4*>(P.PGZ + tb));
        if constexpr (F32) {
#pragma unroll
          for (int p = 0; p < kDepPerLane; ++p) {
            const float z2 = p == 0 ? gz.x : p == 1 ? gz.y : p == 2 ? gz.z : gz.w;
            const float x1 = __fadd_rn(__uint_as_float((unsigned)g[p]), sxf);
            const float y1 = __fadd_rn(__uint_as_float((unsigned)(g[p] >> 32)), syf);
            const bool inb = fabsf(x1) < fHL && fabsf(y1) < fHL;
            boxmask |= (unsigned)inb << p;
            const float ax = __fsub_rn(x1, fgSO);
            const float ay = __fsub_rn(y1, fgSO);
            kxv[p] = __float2int_rn(__fmul_rn(ax, finv));
            kyv[p] = __float2int_rn(__fmul_rn(ay, finv));
            const float ddx = __fsub_rn(__fmul_rn((float)kxv[p], fd), ax);
            const float ddy = __fsub_rn(__fmul_rn((float)kyv[p], fd), ay);
            const float dist = __fadd_rn(__fadd_rn(__fmul_rn(ddx, ddx), __fmul_rn(ddy, ddy)), z2);
            hitmask |= (unsigned)(inb && dist <= fr2) << p;
          }
        } else {
          unsigned undecided = 0;
#pragma unroll
          for (int p = 0; p < kDepPerLane; ++p) {
            const float z2 = p == 0 ? gz.x : p == 1 ? gz.y : p == 2 ? gz.z : gz.w;
            const int vx = (int)(unsigned)g[p] + cx, vy = (int)(unsigned)(g[p] >> 32) + cy;
            const bool in = (unsigned)(vx - 2) <= in_max && (unsigned)(vy - 2) <= in_max;
            const bool near = (unsigned)(vx + 1) <= near_max && (unsigned)(vy + 1) <= near_max;
            const float fx = __fsub_rn(__uint_as_float(((unsigned)vx & low) | 0x4B000000u), centre);
            const float fy = __fsub_rn(__uint_as_float(((unsigned)vy & low) | 0x4B000000u), centre);
            const float d2 = __fmaf_rn(fx, fx, __fmaf_rn(fy, fy, z2));
            const bool hit = in && d2 <= lo2;
            boxmask |= (unsigned)in << p;
            hitmask |= (unsigned)hit << p;
            undecided |= (unsigned)(in ? (!hit && d2 <= hi2) : near) << p;
            kxv[p] = vx;
            kyv[p] = vy;
          }
          if (undecided) {
            // the reference's arithmetic in FP64, each operation rounded on its own, on the track as
            // it was submitted. (Copies of x, y and the z part beside the records, 20 bytes more per
            // deposit, spare a lane the index and a second array: 16 tracks of 1e6 deposits, 2 nm,
            // 23.4 against 24.0 ms, the uneven 2,048-track batch 27.2 and 27.3.)
#pragma unroll
            for (int p = 0; p < kDepPerLane; ++p) {
              if (undecided & (1u << p)) {
                // (axis by axis: the loop around has no registers to spare for three at once)
                const uint32_t src = __ldg(&P.PSRC[tb + p]);
                asm volatile("prefetch.global.L1 [%0];" ::"l"(J.y + src));
                asm volatile("prefetch.global.L1 [%0];" ::"l"(J.z + src));
                double c = st_dadd(J.x[src], cs.sx);
                bool inb = fabs(c) < J.HL;
                c = st_dsub(c, J.gSO);
                double k = lattice_index(c, J.d, J.inv_d);
                const int kx = __double2int_rn(k) << S;
                c = st_dsub(st_dmul(k, J.d), c);
                double dist = st_dmul(c, c);
                c = st_dadd(J.y[src], cs.sy);
                inb = inb && fabs(c) < J.HL;
                c = st_dsub(c, J.gSO);
                k = lattice_index(c, J.d, J.inv_d);
                const int ky = __double2int_rn(k) << S;
                c = st_dsub(st_dmul(k, J.d), c);
                dist = st_dadd(dist, st_dmul(c, c));
                c = st_dsub(st_dadd(J.z[src], J.zsh), J.gSO);
                k = lattice_index(c, J.d, J.inv_d);
                c = st_dsub(st_dmul(k, J.d), c);
                dist = st_dadd(dist, st_dmul(c, c));
                boxmask = (boxmask & ~(1u << p)) | ((unsigned)inb << p);
                hitmask |= (unsigned)(inb && dist <= J.r2) << p;
                kxv[p] = kx;
                kyv[p] = ky;
              }
            }
          }
        }
        if (wins) {  // lane's deposits 4 * lane + 0..3 of the tile that the window holds
          unsigned in = 0xFu;
          if (w == w0) in &= 0xFu << min(max(clip0 - 4 * lane, 0), 4);
          if (w == w1 - 1) in &= (1u << min(max(clip1 - 4 * lane, 0), 4)) - 1u;
          hitmask &= in;
          boxmask &= in;
        }
        hits += __popc(hitmask);
        inbox += __popc(boxmask);
        // runs of equal keys inside the lane's consecutive deposits are summed in registers
        uint64_t rkey = kEmptyKey, rlo = 0, rhi = 0;
        bool rflag = false;
  #pragma unroll
        for (int p = 0; p < kDepPerLane; ++p) {
          if (hitmask & (1u << p)) {
            const int64_t idx = tb + p;
            const ulonglong2 v = __ldg(&P.PV[idx]);
            const uint64_t lo = v.x;
            const uint64_t hi = v.y;
            const uint64_t kzw = __ldg(&P.PKEY[idx]);
            // (the FP32 form converts a lattice index like the reference's llrint: sign-extended)
            const uint64_t key =
                (F32 ? (uint64_t)(int64_t)kxv[p] + (uint64_t)(int64_t)kyv[p] * N
                     : (uint64_t)(uint32_t)(kxv[p] >> S) + (uint64_t)(uint32_t)(kyv[p] >> S) * N) +
                (kzw & ~kBoundaryBit);
            const bool bflag = (kzw & kBoundaryBit) != 0;
            if (key == rkey) {
              add128(rlo, rhi, lo, hi);
              rflag |= bflag;
            } else {
              if (rkey != kEmptyKey) sphere_add<CAP>(T, &cs, P, G, rkey, rlo, rhi, rflag, slot);
              rkey = key; rlo = lo; rhi = hi; rflag = bflag;
            }
          }
        }
        // The lane's last run goes to the table as it is, also when its neighbours hold the same
        // sphere: the 32-bit adds of one slot serialise in shared memory for less than a segmented
        // sum over the warp's lanes costs in shuffles (fused kernel without / with that sum: uneven
        // 2,048-track batch 25.4 / 26.5 ms, single-precision mix 6.8 / 7.1 ms, 2 nm ions
        // 24.9 / 25.4 ms).
        if (rkey != kEmptyKey) sphere_add<CAP>(T, &cs, P, G, rkey, rlo, rhi, rflag, slot);
      }
    }
    if (windowed) {
      // window done: spheres without boundary contributions are complete -> bin them now;
      // the others (or all, if the window overflowed) go to the spill table
      __syncthreads();
      const int cnt = cs.tc[slot];
      if (more && cnt <= CAP / 2) {  // a bin larger than a window, and room for more spheres
        __syncthreads();  // (every thread has read the count)
        continue;
      }
      const bool all_out = cs.ovf[slot] != 0 || more || logged;
      logged = more;
      if (tid == 0) {  // the next window's slot: last read two windows ago
        cs.tc[(wi + 1) % 3] = 0;
        cs.ovf[(wi + 1) % 3] = 0;
      }
      int sent = 0;
      const BinRegs BR(B);
      for (int i = tid; i < cnt; i += THREADS) {
        const uint32_t h = T.used()[i];
        const unsigned bit = 1u << (h & 31);
        const bool flagged = !wins && (T.flags()[h >> 5] & bit) != 0;
        if (flagged) atomicAnd(&T.flags()[h >> 5], ~bit);
        const bool out = all_out || flagged;
        if (out && log_mode) {
          log_append(&cs, P, G, T.keys()[h], T.lo(h), T.hi()[h]);
        } else if (out) {
          if (!gtable_add(G.keys, G.lo, G.hi, G.used, G.count, G.cap, T.keys()[h], T.lo(h), T.hi()[h]))
            atomicOr(P.error_flags, 1);
          sent = 1;
        } else {
          bin_sphere(BR, B, P, [&] { return T.keys()[h]; }, T.lo(h), T.hi()[h], spheres, binned, os);
        }
        T.clear(h);
      }
      // the table and its boundary bits are clear again once every thread is past this point
      sent = __syncthreads_or(sent);
      if (sent && tid == 0) cs.spilled = 1;
    } else if (window_checks && at < end) {
      if (cta_over(&cs.tc[0], P.flush_threshold)) {
        if (log_mode) flush_to_log<CAP, THREADS>(T, cs.tc[0], &cs, P, G);
        else flush_to_spill<CAP, THREADS>(T, cs.tc[0], P, G);
        __syncthreads();
        if (tid == 0) { cs.tc[0] = 0; cs.spilled |= !log_mode; }
        __syncthreads();
      }
    }
    ++wi;
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------------------------
// k_fused: persistent work-stealing kernel. Items are either private (every window of a block of
// oversamples of a small or medium job, one CTA) or helpers of a shared unit (one oversample of
// a large job, whose window chunks are claimed dynamically by every helper that arrives).
// ---------------------------------------------------------------------------------------------
// Adds the shared-memory copies of a histogram to HBM and clears them (all threads of the CTA).
template <int THREADS>
__device__ __forceinline__ void flush_histogram(const HistDev& H, int HB, const double* sedges,
                                                unsigned int* hcount, unsigned long long* hylo,
                                                unsigned long long* hyhi) {
  const int copies = min(kHistCopies, HB / H.nbins);
  for (int b = threadIdx.x; b < H.nbins; b += THREADS) {
    unsigned cnt = 0;
    for (int c = 0; c < copies; ++c) cnt += hcount[c * H.nbins + b];
    if (!cnt) continue;  // nothing in the bin's sums either
    const uint64_t eb = (uint64_t)__double_as_longlong(sedges[b]);
    const bool exact = (int64_t)eb > 0 && (eb >> 52) != 0;  // as in bin_sphere
    uint64_t lo = 0, hi = 0;
    double ys = 0.0;
    for (int c = 0; c < copies; ++c) {
      const int i = c * H.nbins + b;
      if (exact) add128(lo, hi, hylo[i], hyhi[i]);
      else ys += __longlong_as_double((long long)hylo[i]);
      hcount[i] = 0;
      hylo[i] = 0;
      hyhi[i] = 0;
    }
    atomicAdd(&H.counts[b], (unsigned long long)cnt);
    atomicAdd(&H.yfy[b], exact ? from_fixed(lo, hi, (int)(eb >> 52) - 1075) : ys);
  }
}

template <int CAP, int THREADS, bool F32>
__global__ void __launch_bounds__(THREADS, 1) k_fused(FusedParams P) {
  static_assert(CAP <= 65536, "used-slot list stores 16-bit slot indices");
  static_assert(THREADS / 32 == kFusedWarps, "a window is one CTA tile of warp tiles");
  __shared__ CtaState cs;
  __shared__ int s_bcast[2];
  __shared__ BinContext sB;   // the item's binning context and spill table, uniform over the
  __shared__ Spill sG;        // CTA: kept in shared memory rather than in every thread's registers
  __shared__ FusedJob sF;     // (likewise the job)

  const int HB = P.smem_hist_bins;
  const SmemTable<CAP> T;
  unsigned long long* hylo = reinterpret_cast<unsigned long long*>(SmemTable<CAP>::hist());
  unsigned long long* hyhi = hylo + HB;
  double* sedges = reinterpret_cast<double*>(hyhi + HB);         // HB + 1 edges
  unsigned int* hcount = reinterpret_cast<unsigned int*>(sedges + HB + 1);

  const int tid = threadIdx.x;
  const int lane = tid & 31;

  for (int i = tid; i < CAP; i += THREADS) T.clear(i);
  for (int i = tid; i < HB; i += THREADS) { hcount[i] = 0; hylo[i] = 0; hyhi[i] = 0; }
  for (int i = tid; i < CAP / 32; i += THREADS) T.flags()[i] = 0;
  if (tid == 0) {
    for (int k = 0; k < 3; ++k) { cs.tc[k] = 0; cs.ovf[k] = 0; }
    cs.spilled = 0;
    cs.log_mode = 0;
    cs.logn = 0;
    cs.edges_hist = -1;
    cs.table = -1;
    cs.hist_work = 0;
    cs.hist_span = 0;
  }
  __syncthreads();

  for (;;) {
    if (tid == 0) cs.item = (int)atomicAdd(P.work_counter, 1u);
    __syncthreads();
    const int it = cs.item;
    const int cached_hist = cs.edges_hist;
    const long long hist_work = cs.hist_work;
    __syncthreads();
    if (it >= *P.n_items) break;

    const WorkItem W = P.items[it];
    const JobAux A = P.aux[W.job];
    if (A.flags & kAuxNonfinite) continue;  // rejected job: contributes nothing, host reports it
    static_assert(sizeof(JobDev) % 8 == 0, "copied by 64-bit words");
    if (tid < (int)(sizeof(JobDev) / 8))
      reinterpret_cast<unsigned long long*>(&sF.J)[tid] =
          reinterpret_cast<const unsigned long long*>(&P.jobs[W.job])[tid];
    __syncthreads();
    const FusedJob& F = sF;
    const int E0 = choose_grid_exponent(A.e_min, A.e_max, F.J.n, A.flags & kAuxNonzero);
    const int64_t n_wt = (A.kept + kWarpTile - 1) / kWarpTile;
    if (tid == 0) {
      sF.windowed = A.windowed;
      sF.wins = A.windowed == kWinLayers ? P.wins + F.J.win_off : nullptr;
      sF.win_tiles = coarse_windows(F.J, A) ? kCoarseTiles : kWinTiles;
    }
    const HistDev H = P.hists[F.J.hist];
    const bool smem_hist = H.nbins <= HB;

    // the histogram in shared memory: edges and sums stay while consecutive items use the same
    // one (each item fills a bin by at most its own deposit*oversamples: they are added to HBM
    // before the 32-bit counts or the 128-bit sums could wrap, see keep_bits). 64 short tracks on one 3,000-bin spectrum: fused
    // 0.108 ms with a flush per item, 0.089 ms without.
    const int n_os = W.os_count < 0 ? 1 : W.os_count;
    const long long work = A.kept * n_os;
    const bool full = hist_work + work > (1ll << H.keep_bits);
    if (smem_hist && (cached_hist != F.J.hist || full)) {
      if (cached_hist >= 0) {
        flush_histogram<THREADS>(P.hists[cached_hist], HB, sedges, hcount, hylo, hyhi);
        __syncthreads();
      }
      for (int i = tid; i <= H.nbins; i += THREADS) sedges[i] = H.edges[i];
      __syncthreads();
      if (tid == 0) {
        cs.edges_hist = F.J.hist;
        cs.hist_work = 0;
        cs.hist_span = sum_span(H.keep_bits, work);
      }
    }

    if (tid == 0) {
      cs.hist_work += work;
      sB.edges = smem_hist ? sedges : H.edges;
      sB.gcounts = H.counts;
      sB.gyfy = H.yfy;
      sB.nbins = H.nbins;
      sB.mode = H.mode;
      sB.ca = H.ca;
      sB.cb = H.cb;
      sB.E0 = E0;
      sB.scale = E0 > -960 && E0 < 900 ? __longlong_as_double((long long)(E0 + 1023) << 52) : 0.0;
      sB.job = W.job;
      sB.span = cs.hist_span;
      sB.hcount = smem_hist ? hcount : nullptr;
      sB.hylo = smem_hist ? hylo : nullptr;
      sB.hyhi = smem_hist ? hyhi : nullptr;
      sB.copies = smem_hist ? min(kHistCopies, HB / H.nbins) : 1;
    }
    __syncthreads();
    const BinContext& B = sB;

    // per-thread counts of one item (an item covers at most a few million deposit*oversamples)
    unsigned int hits = 0, spheres = 0, binned = 0, inbox = 0;

    // Segments: a private item walks its oversamples (all windows each) with one pool table; a
    // helper claims window chunks of its shared unit until none is left.
    const bool shared = W.unit >= 0;
    const int64_t wpc = chunk_tiles(P.chunk_windows);  // warp tiles per chunk
    const int64_t n_chunks = (n_wt + wpc - 1) / wpc;
    // A private item's spill table stays with the CTA for its next private items; it goes back to
    // the pool before the CTA joins a shared unit, so that a CTA holds at most one.
    if (tid == 0) {
      if (!shared && cs.table < 0) {
        cs.table = pool_acquire(P.pool_bits, gridDim.x, P.error_flags);
      } else if (shared && cs.table >= 0) {
        __threadfence();
        pool_release(P.pool_bits, cs.table);
        cs.table = -1;
      }
    }
    __syncthreads();
    const int private_table = cs.table;
    for (int seg = 0;; ++seg) {
      int os, t;
      int64_t wb, we;
      if (!shared) {
        if (private_table < 0 || seg >= n_os) break;
        os = W.os_begin + seg;
        t = private_table;
        wb = 0;
        we = n_wt;
        if (F.wins) {
          // whole bins: a window that continues a bin belongs to the item that began it
          wb = W.os_count < 0 ? (int64_t)(-1 - W.unit) * -W.os_count : 0;
          we = W.os_count < 0 ? min(wb - W.os_count, (int64_t)A.n_win) : (int64_t)A.n_win;
          while (wb < A.n_win && (F.wins[wb] & kWinContinues)) ++wb;
          while (we < A.n_win && (F.wins[we] & kWinContinues)) ++we;
        }
      } else {
        if (tid == 0) {
          const unsigned c = atomicAdd(&P.unit_next[W.unit], 1u);
          s_bcast[0] = (int64_t)c < n_chunks ? (int)c : -1;
          s_bcast[1] = s_bcast[0] >= 0 ? unit_table_get(P, W.unit) : -1;
        }
        __syncthreads();
        const int c = s_bcast[0];
        t = s_bcast[1];
        __syncthreads();
        if (c < 0 || t < 0) break;
        os = W.os_begin;
        wb = (int64_t)c * wpc;
        we = wb + wpc < n_wt ? wb + wpc : n_wt;
      }
      if (tid == 0) {
        sG = spill_of(P, t, A.kept);
        cs.log_mode = !shared;  // a single CTA sees every window of the oversample
        const JobDev& J = F.J;
        float ux, uy;
        shift_uniforms(J.seed, J.track_id, (uint32_t)os, J.shift_track, &ux, &uy);
        cs.sx = shift_from_uniform(ux, J.L, J.HL);
        cs.sy = shift_from_uniform(uy, J.L, J.HL);
        const int half = 1 << J.g_shift >> 1;
        cs.cx = __double2int_rn(st_dmul(st_dsub(cs.sx, J.gSO), J.g_scale)) + half;
        cs.cy = __double2int_rn(st_dmul(st_dsub(cs.sy, J.gSO), J.g_scale)) + half;
      }
      __syncthreads();
      const Spill& G = sG;
      superimpose<CAP, THREADS, F32>(P, F, T, cs, G, B, os, wb, we, hits, inbox, spheres, binned);
      if (cs.log_mode) {
        if (!F.windowed && cs.logn > 0) {
          // the table's spheres may have parts in the log: they join it
          flush_to_log<CAP, THREADS>(T, cs.tc[0], &cs, P, G);
          __syncthreads();
          if (tid == 0) cs.tc[0] = 0;
          __syncthreads();
        }
        log_reduce<CAP, THREADS>(T, cs, P, G, B, spheres, binned, os);
      }
      const int cnt = F.windowed ? 0 : cs.tc[0];  // flagged windows leave the table empty
      bool bin_table;
      if (!shared) {
        bin_table = cs.spilled != 0;
        if (bin_table) {
          flush_to_spill<CAP, THREADS>(T, cnt, P, G);
        } else {
          const BinRegs BR(B);
          for (int i = tid; i < cnt; i += THREADS) {
            const uint32_t h = T.used()[i];
            bin_sphere(BR, B, P, [&] { return T.keys()[h]; }, T.lo(h), T.hi()[h], spheres, binned, os);
            T.clear(h);
          }
        }
        __syncthreads();
      } else {
        // everything left in shared memory may meet contributions of other chunks
        flush_to_spill<CAP, THREADS>(T, cnt, P, G);
        __threadfence();
        __syncthreads();
        if (tid == 0) {
          const unsigned done = atomicAdd(&P.unit_done[W.unit], 1u) + 1u;
          s_bcast[0] = (int64_t)done == n_chunks ? 1 : 0;
        }
        __syncthreads();
        bin_table = s_bcast[0] != 0;  // last chunk of the unit: every contribution is in G
        if (bin_table) __threadfence();
      }
      if (bin_table) {
        bin_spill<THREADS>(G, B, P, spheres, binned, os);
        if (shared && tid == 0) pool_release(P.pool_bits, t);
      }
      if (tid == 0) {
        for (int k = 0; k < 3; ++k) { cs.tc[k] = 0; cs.ovf[k] = 0; }
        cs.spilled = 0;
        cs.log_mode = 0;
      }
      __syncthreads();
    }
    unsigned long long w_hits = hits, w_spheres = spheres, w_binned = binned, w_inbox = inbox;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      w_hits += __shfl_xor_sync(0xffffffffu, w_hits, o);
      w_spheres += __shfl_xor_sync(0xffffffffu, w_spheres, o);
      w_binned += __shfl_xor_sync(0xffffffffu, w_binned, o);
      w_inbox += __shfl_xor_sync(0xffffffffu, w_inbox, o);
    }
    if (lane == 0) {
      if (w_hits) atomicAdd(&P.aux[W.job].hits, w_hits);
      if (w_spheres) atomicAdd(&P.aux[W.job].spheres, w_spheres);
      if (w_binned) atomicAdd(&P.aux[W.job].binned, w_binned);
      if (w_inbox) atomicAdd(&P.aux[W.job].inbox, w_inbox);
    }
    __syncthreads();
  }
  if (cs.edges_hist >= 0)
    flush_histogram<THREADS>(P.hists[cs.edges_hist], HB, sedges, hcount, hylo, hyhi);
}

// The run's state on the device to its initial values. One kernel rather than a memset per array: ten
// operations in a row cost a small batch more than its superimposition; and no copy from the host:
// a host-to-device copy on the run's stream would queue on a copy engine behind any track upload in
// flight and hold the run's kernels back.
__global__ void __launch_bounds__(256) k_reset(const __grid_constant__ ResetParams p) {
  cudaTriggerProgrammaticLaunchCompletion();
  const int64_t i0 = (int64_t)blockIdx.x * 256 + threadIdx.x, step = (int64_t)gridDim.x * 256;
  for (int64_t j = i0; j < p.n_jobs; j += step) {
    JobAux a = {};
    a.e_min = INT_MAX;
    a.e_max = INT_MIN;
    p.aux[j] = a;
  }
  for (int64_t i = i0; i < p.n_units; i += step) {
    p.u_next[i] = 0;
    p.u_done[i] = 0;
    p.u_table[i] = ~0u;
  }
  for (int64_t i = i0; i < p.n_bins; i += step) p.bins[i] = 0;
  for (int64_t i = i0; i < p.n_pool; i += step) p.pool[i] = 0;
  for (int64_t i = i0; i < kPlanScratch / 4; i += step) p.plan[i] = 0;
  if (i0 < 4) {
    p.counter[i0] = 0;
    if (p.err) p.err[i0] = 0;
    if (p.ex_count) p.ex_count[i0] = 0;
  }
  if (p.gkeys) {
    for (int64_t i = i0; i < p.n_slots; i += step) {
      p.gkeys[i] = kEmptyKey;
      p.glo[i] = 0;
      p.ghi[i] = 0;
    }
    for (int64_t i = i0; i < p.n_tables; i += step) p.gcount[i] = 0;
  }
}

// Launches a kernel; `chained` when another kernel of this file is directly before it on the stream
// (no event or copy between): it is then launched without waiting for that one to drain, and its
// CTAs, placed meanwhile, wait in chain_start. A chained kernel's CTAs are placed only after every
// CTA of the one before has started, so they take no place that it still needs. What the launch
// latency of each kernel in a row cost small batches (per pass, plain / chained): the call without
// allocation 100 / 91 us, one proton track of 19,997 deposits 183 / 168 us, 16 short tracks one at a
// time 1.68 / 1.56 ms; runs replayed as graphs and large batches stay as they are.
template <typename P>
static void launch_chained(void (*kernel)(P), unsigned blocks, unsigned threads, cudaStream_t s,
                           bool chained, const P& p) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(threads);
  cfg.stream = s;
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = chained ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, p);
}

cudaError_t launch_reset(const ResetParams& p, cudaStream_t s) {
  int64_t most = p.n_jobs > p.n_units ? p.n_jobs : p.n_units;
  if (p.n_bins > most) most = p.n_bins;
  if (p.gkeys && p.n_slots > most) most = p.n_slots;
  const int64_t blocks = (most + 255) / 256;
  k_reset<<<(unsigned)(blocks < 1 ? 1 : blocks > 592 ? 592 : blocks), 256, 0, s>>>(p);
  return cudaGetLastError();
}

int plan_launches(int n_jobs) { return n_jobs <= 0 ? 0 : n_jobs > kPlanSmall ? 2 : 1; }

cudaError_t launch_plan(const PlanParams& q, bool chained, cudaStream_t s) {
  if (q.n_jobs <= 0) return cudaSuccess;
  launch_chained(k_plan, 1u, 1024u, s, chained, q);
  if (q.n_jobs > kPlanSmall) launch_chained(k_plan_write, (unsigned)q.n_jobs, 128u, s, true, q);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// FP64 issue-rate probe: independent chains of dependent double additions and multiplications
// (8 chains per thread), used to measure the FP64 pipe throughput the fused kernel is bound by.
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_fp64_probe(double* out, int iters, double a, double b) {
  double v[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) v[k] = (double)(threadIdx.x + k) * 1e-3;
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = __dadd_rn(__dmul_rn(v[k], a), b);
  }
  double s = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) s += v[k];
  if (s == 12345.678) out[blockIdx.x] = s;  // keeps the chains alive
}

// One helper's wait for the table of shared unit 0 (unit_table_get), with max_polls sleeps;
// out[0] receives the table it got (-1: the wait ran out).
__global__ void k_unit_wait_probe(FusedParams p, long long max_polls, int* out) {
  if (threadIdx.x == 0 && blockIdx.x == 0) out[0] = unit_table_get(p, 0, max_polls);
}

cudaError_t launch_unit_wait_probe(int* table, int* error_flags, int* out, long long max_polls,
                                   cudaStream_t s) {
  FusedParams p{};
  p.unit_table = table;
  p.error_flags = error_flags;
  k_unit_wait_probe<<<1, 32, 0, s>>>(p, max_polls, out);
  return cudaGetLastError();
}

cudaError_t launch_fp64_probe(double* out, int blocks, int iters, cudaStream_t s) {
  k_fp64_probe<<<blocks, 256, 0, s>>>(out, iters, 0.999999999, 1e-9);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Shared-memory atomic probe: 64-bit atomic additions on a 4096-slot shared array, one CTA of
// 1024 threads per SM (the fused kernel's shape). The lanes of a warp update consecutive slots
// (no bank conflict beyond the two wavefronts a 64-bit warp access needs), so the rate is the
// peak the fused kernel's per-hit and per-sphere shared-memory updates are set against.
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(1024, 1) k_smem_atomic_probe(unsigned long long* out, int iters) {
  __shared__ unsigned long long s[4096];
  for (int i = threadIdx.x; i < 4096; i += blockDim.x) s[i] = 0;
  __syncthreads();
  const unsigned idx = threadIdx.x;  // 1024 distinct slots: lanes of a warp are consecutive
  for (int i = 0; i < iters; ++i) atomicAdd(&s[(idx + (unsigned)i * 1024u) & 4095u], 1ull);
  __syncthreads();
  if (threadIdx.x == 0) out[blockIdx.x] = s[0] + s[4095];
}

cudaError_t launch_smem_atomic_probe(unsigned long long* out, int blocks, int iters, cudaStream_t s) {
  k_smem_atomic_probe<<<blocks, 1024, 0, s>>>(out, iters);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Host-side launch wrappers
// ---------------------------------------------------------------------------------------------
// 32 warps (64 registers each): the kernel is latency-bound, and more resident warps hide more
// of it than longer per-thread blocks would.
constexpr int kFusedThreads = 1024;

// Two shapes of the fused kernel: a 4096-slot sphere table with room for histograms of up to
// 4096 bins in shared memory, or an 8192-slot table when every histogram of the batch has at
// most kSmallHistBins bins.
constexpr int kSmallHistBins = 600;
constexpr int kBigHistBins = 4096;

bool fused_big_table(int max_nbins, int table_slots) {
  return max_nbins <= kSmallHistBins && table_slots != 4096;
}

size_t fused_smem_bytes(int cap, int hist_bins) {
  return (size_t)cap * 26 + (size_t)cap / 8 + (size_t)hist_bins * 28 + 8;
}

int prepare_launches(int64_t n_blocks, bool any_flagged) {
  return n_blocks <= 0 ? 0 : any_flagged ? 6 : 4;
}

cudaError_t launch_prepare(const PrepareParams& p, int64_t n_blocks, bool any_flagged,
                           bool chained, cudaStream_t s) {
  if (n_blocks <= 0) return cudaSuccess;
  const unsigned blocks = (unsigned)n_blocks, jobs = (unsigned)p.n_jobs;
  launch_chained(k_prep_count, blocks, kPrepThreads, s, chained, p);
  launch_chained(k_prep_scan, jobs, 1024, s, true, p);
  if (any_flagged) launch_chained(k_prep_cells, 592, kPrepThreads, s, true, p);
  launch_chained(k_prep_write, blocks, kPrepThreads, s, true, p);
  launch_chained(k_prep_pad, jobs, kWarpTile, s, true, p);
  if (any_flagged) launch_chained(k_prep_flag, blocks, kPrepThreads, s, true, p);
  return cudaGetLastError();
}

template <bool F32>
static cudaError_t configure_fused_form() {
  cudaError_t e = cudaFuncSetAttribute(k_fused<4096, kFusedThreads, F32>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)fused_smem_bytes(4096, kBigHistBins));
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(k_fused<8192, kFusedThreads, F32>,
                              cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)fused_smem_bytes(8192, kSmallHistBins));
}

cudaError_t configure_fused() {
  const cudaError_t e = configure_fused_form<false>();
  return e != cudaSuccess ? e : configure_fused_form<true>();
}

template <bool F32>
static void launch_fused_form(const FusedParams& p, int grid, bool big_table, cudaStream_t s) {
  if (big_table)
    k_fused<8192, kFusedThreads, F32>
        <<<grid, kFusedThreads, fused_smem_bytes(8192, kSmallHistBins), s>>>(p);
  else
    k_fused<4096, kFusedThreads, F32>
        <<<grid, kFusedThreads, fused_smem_bytes(4096, kBigHistBins), s>>>(p);
}

// Picks the kernel shape: the 8192-slot sphere table when the largest histogram of the batch
// fits the remaining shared memory (and table_slots does not ask for 4096), else 4096 slots with
// room for 4096 bins; fills P.smem_hist_bins and P.flush_threshold. P.fp32 picks the FP32
// geometry form.
cudaError_t launch_fused(FusedParams p, int max_nbins, int grid, int table_slots, cudaStream_t s) {
  if (grid <= 0) return cudaSuccess;
  const bool big_table = fused_big_table(max_nbins, table_slots);
  if (big_table) {
    p.smem_hist_bins = kSmallHistBins;
    p.flush_threshold = 8192 - 4096 - 8192 / 4;  // unused: no window checks on this table
  } else {
    p.smem_hist_bins = kBigHistBins;
    p.flush_threshold = 4096 / 2;
  }
  if (p.fp32) launch_fused_form<true>(p, grid, big_table, s);
  else launch_fused_form<false>(p, grid, big_table, s);
  return cudaGetLastError();
}

int fused_threads() { return kFusedThreads; }

}  // namespace st
