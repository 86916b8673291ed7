// The grid build as four launches (fs_grid.cu holds the two in the middle):
//   1. keys     cell key and arrival slot of every particle, the occupancy of
//               every cell and of every tile of 4,096 cells (atomics, a
//               block's tiles counted in shared memory first); the positions
//               come from a Key functor, so that a substep's predict or
//               integrate step runs here instead of in a pass of its own
//   2. scan     exclusive prefix of the occupancies: each tile adds up the
//               sums of the tiles before it, scans its cells and clears the
//               counts it found for the next build
//   3. scatter  tmp[off[key] + arrival] = i; clears the tile sums (so both are
//               zero between builds, with no memset)
//   4. rank     the stable order inside each cell (ascending ids), and a
//               Gather functor that copies what the neighbour loops read into
//               cell order while the particle's index and slot are at hand
// What bounds it: at small counts the launches and the 16.8 MB that the scan
// of 128^3 cells moves through L2, at large ones the scattered accesses of
// keys and rank.  B200, predict + build + gather of a PBF substep: 35 + 9 + 7
// us in eleven launches before, 22 in these four at 4,079 particles; 45 + 19 +
// 13 and 48 at 401,856.
#pragma once

#include "fs_nbr.cuh"
#include "fs_sort.cuh"

namespace fs {

constexpr int kRankThreads = 512;
constexpr int kScanThreads = 512;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;  // 4096 cells per tile

struct KeyArgs {
  GridDev g;               // dims, rounding, worlds, inv of this build
  const int32_t* world;    // particle_world (batched contexts)
  int32_t discard;         // key of non-finite positions
  int32_t *key, *slot, *count, *tile_sum;
  int32_t ntiles, copies;  // tile_sum[copies][ntiles]
  uint32_t* status;
  ListCtl* ctl;
  const fs_frame_clock* clock;
};

// Key functors: reset() runs once per launch before anything else (even when
// the frame clock is idle); position(t, i) returns the position to bin of the
// particle that thread t takes, and its index i.
struct KeyPositions {
  const float* x;
  FS_DEV void reset() const {}
  FS_DEV float3 position(int64_t t, int64_t& i) const {
    i = t;
    return ld3(x, t);
  }
};

struct NoGather {
  FS_DEV void operator()(int64_t, int32_t) const {}
};

// What the neighbour loops read (gather_common_slot).
struct CommonGather {
  fs_model m;
  const float *x, *v;
  float4* xs;
  ScanOut q;
  float4* vs;
  float *mv, *ms;
  uint32_t* status;
  int nworlds;
  FS_DEV void operator()(int64_t s, int32_t i) const {
    gather_common_slot(s, i, m, x, v, xs, q, vs, mv, ms, status, nworlds);
  }
};

template <class Key>
__global__ void k_cell_keys(int64_t n, Key source, KeyArgs a) {
  grid_begin();
  const int64_t t = thread_id();
  if (t == 0) {
    source.reset();
    *a.ctl = ListCtl{};  // a new grid invalidates recorded neighbour lists
  }
  if (clock_idle(a.clock)) return;
  // Lattice-ordered particles run along z, whose cells lie tiles apart: every
  // block meets the same hundred tiles.  One global atomic per block and tile,
  // spread over a few copies of the sums (at 1,000,003 particles the kernel
  // took 94 us with an atomic per warp and tile, 48 with one copy).
  extern __shared__ int32_t tile[];
  for (int k = threadIdx.x; k < a.ntiles; k += blockDim.x) tile[k] = 0;
  __syncthreads();
  if (t < n) {
    int64_t i;
    const float3 p = source.position(t, i);
    int k = a.discard;
    if (a.g.worlds) {
      const int w = a.world[i];
      if (w < 0 || w >= a.g.nworlds) atomicOr(a.status, FS_STATUS_BOUNDS);
      if (isfinite(p.x) && isfinite(p.y) && isfinite(p.z))
        k = world_cell_key(a.g.worlds[world_index(w, a.g.nworlds)], a.g.inv, p.x, p.y, p.z);
    } else if (isfinite(p.x) && isfinite(p.y) && isfinite(p.z)) {
      k = phys_cell(a.g, to_cell(__fmul_rn(p.x, a.g.inv), a.g.rounding), to_cell(__fmul_rn(p.y, a.g.inv), a.g.rounding),
                    to_cell(__fmul_rn(p.z, a.g.inv), a.g.rounding));
    }
    if (k == a.discard) atomicOr(a.status, FS_STATUS_NONFINITE);
    a.key[i] = k;
    a.slot[i] = atomicAdd(a.count + k, 1);
    atomicAdd(tile + k / kScanTile, 1);
  }
  __syncthreads();
  int32_t* const sum = a.tile_sum + (blockIdx.x % a.copies) * a.ntiles;
  for (int k = threadIdx.x; k < a.ntiles; k += blockDim.x)
    if (tile[k]) atomicAdd(sum + k, tile[k]);
}

// Slot of particle i = tmp[s] inside its cell, by counting the smaller ids of
// the cell (up to kSmallCell of them); a more crowded cell is sorted by the
// block that holds its first slot.  32 registers (four blocks an SM): at the 40
// that the sort would take, builds of 1,000,003 particles went from 50.0 to
// 52.2 us and the WCSPH substep of 4,194,304 from 1,855 to 1,881.
template <class Gather>
__global__ void __launch_bounds__(kRankThreads, 4) k_rank(int64_t n, const int32_t* __restrict__ key,
                                                       const int32_t* __restrict__ off,
                                                       const int32_t* __restrict__ tmp, int32_t* perm,
                                                       Gather gather, const fs_frame_clock* clock) {
  __shared__ int32_t smem[kSortSmemInts];
  __shared__ int32_t crowded[kRankThreads / kSmallCell + 1];
  __shared__ int ncrowded;
  grid_begin();
  if (clock_idle(clock)) return;
  if (threadIdx.x == 0) ncrowded = 0;
  __syncthreads();
  const int64_t s = thread_id();
  if (s < n) {
    const int32_t i = tmp[s];
    const int32_t c = key[i];
    const int32_t a = off[c], b = off[c + 1];
    if (b - a > kSmallCell) {
      if (s == a) crowded[atomicAdd(&ncrowded, 1)] = c;
    } else {
      int32_t slot = a;
      for (int32_t t = a; t < b; ++t) slot += tmp[t] < i ? 1 : 0;
      perm[slot] = i;
      gather(slot, i);
    }
  }
  __syncthreads();
  const int nc = ncrowded;
  for (int k = 0; k < nc; ++k) {
    const int32_t c = crowded[k];
    const int32_t a = off[c], len = off[c + 1] - a;
    block_sort_ids(tmp + a, perm + a, len, n, smem);
    for (int j = threadIdx.x; j < len; j += blockDim.x) gather(a + j, perm[a + j]);
    __syncthreads();
  }
}

// fs_grid.cu: argument checks, the arguments of the first launch and the
// context's note that a build has begun; the scan and the scatter; the note of
// the finished build (launched: what its launches returned).
//
// Each launch of a build writes where the one before it says: with the offsets
// of an earlier build, or with counts that a scan has not cleared, the scatter
// would write past its array.  So the first launch that fails ends the build,
// and the next build clears the counts before it counts.
int grid_prepare(fs_context* c, int64_t n, float radius, cudaStream_t st, const int32_t* world,
                 const fs_frame_clock* clock, KeyArgs* a);
cudaError_t grid_scan_scatter(fs_context* c, int64_t n, cudaStream_t st, const fs_frame_clock* clock);
int grid_finish(fs_context* c, int64_t n, float radius, cudaStream_t st, cudaError_t launched);

// Builds the grid of n > 0 positions of the Key functor and gathers into cell
// order.  world: particle_world (required by batched contexts).  clock
// (optional): a device-side frame clock; nothing is done while it is idle.
template <class Key, class Gather>
int grid_build(fs_context* c, int64_t n, float radius, cudaStream_t st, const int32_t* world,
               const fs_frame_clock* clock, const Key& source, const Gather& gather) {
  KeyArgs a;
  int rc = grid_prepare(c, n, radius, st, world, clock, &a);
  if (rc) return rc;
  PassScope ps_(c, P_GRID, st, 4);
  cudaError_t e = launch(k_cell_keys<Key>, blocks_for(n), kBlock, sizeof(int32_t) * a.ntiles, st, n, source, a);
  if (!e) e = grid_scan_scatter(c, n, st, clock);
  if (!e)
    e = launch(k_rank<Gather>, blocks_for(n, kRankThreads), kRankThreads, 0, st, n, c->key, c->cell_off, c->tmp_ids,
               c->perm, gather, clock);
  return grid_finish(c, n, radius, st, e);
}

}  // namespace fs
