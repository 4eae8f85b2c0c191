// cluster.cuh -- Euclidean cluster roots on the radius grid.
//
// The component structure of "dx*dx + dy*dy + dz*dz <= tol*tol" (f32, the
// predicate of uniform_grid.rs:440-520 and kdtree.rs:544-549) is unique, and
// so is the reference's answer for each point: the smallest point index of
// its component (union_min_root, uniform_grid.rs:410-418; compress_roots,
// :389-395).  Here the grid of the normal estimator (cell sort, cell table,
// column hash, 3x3 column ranges) supplies the candidates, and a lock-free
// union-find links the pairs.  A root only ever hooks under a smaller one, by
// compare-and-swap on its own word, so every tree's root is the smallest index
// of its points.
//
// Two forests, chosen by the points per occupied cell (cluster_dense):
//
//   over point indices, 32-bit parents: one pass over the pairs, each joined root to
//   root.  Its words take the least memory and traffic, and a pair costs two walks
//   from the points themselves: the cheapest where a point has a pair or less.
//
//   over cell-sorted positions: the node of position i is the word link[i] =
//   (index of its parent point << 32) | position of its parent, so a warp's
//   neighbours share sectors, where a forest over point indices costs a sector of
//   its own for every neighbour, and the index in the high half orders the roots.
//   A sampled pass joins most points of a component through at most five pairs
//   each (the neighbour sampling of Afforest, Sutton et al. 2018), a flattening
//   links every point straight to its root, and then nearly every pair of the full
//   pass hangs under one root and costs one load and a comparison.
#pragma once

#include "normals.cuh"

namespace srcu {

constexpr int CL_THREADS = 256;

// Points per occupied cell from which on the position forest is taken: 1.2, or 1.75
// above CL_LARGE points, where its words and the candidates no longer stay in L2 beside
// the ranges.  Below the line it pays a second walk over the candidates that finds
// little; above it, once the points hang together, the index forest climbs to one far
// root for every pair.  The cluster kernels over indices / over positions, us:
//   scans in random order   100k at 1.09 36 / 42, at 1.54 84 / 67; 500k at 1.15 71 / 79,
//     at 1.35 104 / 100, at 2.07 624 / 151; 1M at 1.17 101 / 133, at 1.31 153 / 145, at
//     1.76 325 / 198; 2M at 1.34 237 / 265, at 1.63 357 / 405, at 2.02 980 / 405; 3M at
//     1.50 393 / 589, at 1.96 1096 / 668
//   along flight lines      1M at 1.31 156 / 152, at 1.51 203 / 219; 2M at 1.63 386 / 429;
//     3M at 1.96 822 / 745, at 3.22 1710 / 886
//   a 131k-point LiDAR frame at 1.58 123 / 98, at 2.33 530 / 276; spheres, planes and
//     cylinders, 500k at 1.38 181 / 116
constexpr uint64_t CL_LARGE = 1536 << 10;
__device__ __forceinline__ bool cluster_dense(const Control *ctl) {
  const uint64_t n = ctl->n_points, cells = ctl->n_cells;
  return n > CL_LARGE ? 4 * n >= 7 * cells : 5 * n >= 6 * cells;
}

// ---- the forest over point indices ---------------------------------------------

// Root of x with path halving.  Parents only ever move to ancestors, so the
// halving writes race benignly with other finds and with the hooks (a hook
// only rewrites the parent word of a root, which this never writes).
__device__ __forceinline__ uint32_t uf_find(uint32_t *parent, uint32_t x, uint32_t *status) {
  for (uint32_t it = 0; it < SPIN_LIMIT; ++it) {
    const uint32_t p = ld_relaxed_u32(parent + x);
    if (p == x) return x;
    const uint32_t gp = ld_relaxed_u32(parent + p);
    if (gp != p) st_relaxed_u32(parent + x, gp);
    x = gp;
  }
  atomicOr(status, ST_TIMEOUT);
  return x;
}

__device__ __forceinline__ void uf_union(uint32_t *parent, uint32_t a, uint32_t b,
                                         uint32_t *status) {
  for (uint32_t it = 0; it < SPIN_LIMIT; ++it) {
    uint32_t ra = uf_find(parent, a, status), rb = uf_find(parent, b, status);
    if (ra == rb) return;
    if (ra > rb) {
      const uint32_t t = ra;
      ra = rb;
      rb = t;
    }
    // hook the larger root under the smaller one; a failed swap means rb
    // stopped being a root meanwhile, so both roots are looked up again
    if (atomicCAS(parent + rb, rb, ra) == rb) return;
  }
  atomicOr(status, ST_TIMEOUT);
}

// ---- the forest over cell-sorted positions -------------------------------------

__device__ __forceinline__ uint64_t uf_word(uint32_t index, uint32_t pos) {
  return (uint64_t(index) << 32) | pos;
}

// Joins the trees of nodes i and j, whose links were a and b, and returns the
// common ancestor found, or UF_NONE after LIMIT steps.  Always the larger word climbs
// (Rem's algorithm: words fall along every path), and a root that is the larger hooks
// under the other by compare-and-swap, root or not; a swap that fails returns the link
// to climb instead.  So the smaller root -- the one nearly every join meets
// once a component has formed -- is never loaded.  On the way up links are halved:
// they only ever move to ancestors, so this races benignly with other walks and
// with the hooks, which rewrite the words of roots alone.
constexpr uint64_t UF_NONE = ~0ull;  // no word: point indices stay below 2^30
template <uint32_t LIMIT>
__device__ __forceinline__ uint64_t uf_join(uint64_t *link, uint32_t i, uint64_t a, uint32_t j,
                                            uint64_t b) {
  for (uint32_t it = 0; it < LIMIT; ++it) {
    if (a == b) return a;
    if (a < b) {
      const uint64_t t = a;
      a = b;
      b = t;
      const uint32_t k = i;
      i = j;
      j = k;
    }
    const uint32_t pos = uint32_t(a);
    uint64_t up = ld_relaxed(link + pos);
    if (up == a) {
      up = atomicCAS(reinterpret_cast<unsigned long long *>(link + pos), a, b);
      if (up == a) return b;
    }
    if (pos != i) st_relaxed(link + i, up);
    i = pos;
    a = up;
  }
  return UF_NONE;
}

// Steps a join of the sampled pass climbs before it leaves the pair to the full pass,
// which meets flattened trees.  Without a limit a lane can climb alone over the links
// that a whole wave has just made: 2M points along a line, its even ones numbered
// before its odd ones, took 235 ms, 200 us so (the index forest: 410 us).  The scans
// gain from it as well: 2M points at 2.5 per cell 525 -> 430 us.
constexpr uint32_t CL_CLIMB = 16;
constexpr uint32_t CL_LOOK = 32;
constexpr uint32_t CL_STEP = 4;

// ---- kernels -------------------------------------------------------------------

// Every point a tree of its own.  The forest's memory holds a 64-bit word per point;
// the index forest uses the first half of it.
__global__ void __launch_bounds__(CL_THREADS) k_cluster_init(Control *ctl, const float4 *pts,
                                                             uint64_t *link) {
  if (ld_relaxed_u32(&ctl->status)) return;
  const uint32_t n = uint32_t(ctl->n_points);
  const bool dense = cluster_dense(ctl);
  uint32_t *parent = reinterpret_cast<uint32_t *>(link);
  for (uint32_t i = blockIdx.x * CL_THREADS + threadIdx.x; i < n; i += gridDim.x * CL_THREADS) {
    if (dense) link[i] = uf_word(__float_as_uint(pts[i].w), i);
    else parent[i] = i;
  }
}

// One lane per cell-sorted point i: the candidates j > i of its 27-cell
// neighbourhood (each unordered pair once) that pass the predicate are joined
// with it -- all of them, or with Sample only the first of each column, sought among
// its first CL_LOOK.  The
// columns before the query's own in key order hold no position above i, so
// the walk starts at its own column (range 4).  The index forest has no sampled pass.
//
// Where a range of the warp is longer than CL_LOOK its lanes walk in step, CL_STEP
// candidates between votes: once a join has parted them they walk the rest of a range
// one after another, which long ranges with few hits make most of (100k points with an
// outlier that widens the cells to 400 points: 10.3 ms, 0.94 so; 1M points at 50 a cell
// 3.8 ms, 1.6 so).  Short ranges, where the votes cost more than they give, go without.
//
// A lane whose point and candidate hang under different words climbs by
// dependent loads from L2 while its warp waits, so the cost is the number of
// such pairs, not the walk.  On a 2M-point scan at tolerance 0.3 (2.5 points per
// cell) all kernels of the position forest take 430 us, 1020 us with the full pass
// alone, and the index forest 1430 us.
template <bool Sample>
__global__ void __launch_bounds__(CL_THREADS) k_cluster_union(Control *ctl, const float4 *pts,
                                                              const uint32_t *pt_cell,
                                                              const uint2 *ranges, float r2,
                                                              uint64_t *link) {
  if (ld_relaxed_u32(&ctl->status)) return;
  const bool dense = cluster_dense(ctl);
  if (Sample && !dense) return;
  const uint32_t n = uint32_t(ctl->n_points);
  const uint64_t u_count = ctl->n_cells;
  uint32_t *parent = reinterpret_cast<uint32_t *>(link);
  const uint32_t lane = threadIdx.x & 31u;
  for (uint32_t base = blockIdx.x * CL_THREADS + (threadIdx.x - lane); base < n;
       base += gridDim.x * CL_THREADS) {
    const uint32_t i = min(base + lane, n - 1);
    const float4 q = pts[i];
    const uint32_t u = pt_cell[i];
    const uint32_t a = __float_as_uint(q.w);
    bool active = base + lane < n;  // the other lanes stay for the warp's votes
    if (u >= u_count || a >= n) {  // cannot happen for a consistent cell table
      atomicOr(&ctl->status, ST_INTERNAL);
      active = false;
    }
    // a NaN coordinate is near nothing, and all of a cloud's NaN points share one cell
    if (isnan(q.x) || isnan(q.y) || isnan(q.z)) active = false;
    const uint2 *rg = active ? ranges + size_t(u) * 9 : nm_no_ranges;
    uint64_t root = dense ? ld_relaxed(link + i) : 0;  // the highest ancestor of i met so far
    auto near = [&](uint32_t j) {
      const float4 c = __ldg(pts + j);
      const float dx = __fsub_rn(c.x, q.x);
      const float dy = __fsub_rn(c.y, q.y);
      const float dz = __fsub_rn(c.z, q.z);
      return __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz)) <= r2;
    };
    auto join = [&](uint32_t j) {
      if (Sample || dense) {
        const uint64_t w = ld_relaxed(link + j);
        if (w == root) return;
        const uint64_t up = uf_join<Sample ? CL_CLIMB : SPIN_LIMIT>(link, i, root, j, w);
        if (up != UF_NONE) root = up;
        else if (!Sample) atomicOr(&ctl->status, ST_TIMEOUT);
      } else {
        const uint32_t b = __float_as_uint(pts[j].w);
        if (b < n) uf_union(parent, a, b, &ctl->status);
        else atomicOr(&ctl->status, ST_INTERNAL);
      }
    };
#pragma unroll 1
    for (int r = 4; r < 9; ++r) {
      const uint2 range = rg[r];
      uint32_t j = max(range.x, i + 1), end = range.y;
      const bool in_step = dense && __any_sync(FULL_MASK, end > j + CL_LOOK);
      if (Sample) end = min(end, j + CL_LOOK);
      if (!in_step) {
        for (; j < end; ++j)
          if (near(j)) {
            join(j);
            if (Sample) break;
          }
        continue;
      }
      for (; __any_sync(FULL_MASK, j < end); j += CL_STEP) {
        uint32_t hits = 0;
#pragma unroll
        for (uint32_t k = 0; k < CL_STEP; ++k)
          if (j + k < end && near(j + k)) hits |= 1u << k;
        if (Sample && hits) {
          hits &= 0u - hits;  // the first
          end = 0;
        }
        if (!__any_sync(FULL_MASK, hits != 0)) continue;
#pragma unroll 1
        for (uint32_t k = 0; k < CL_STEP; ++k) {
          if ((hits >> k) & 1u) join(j + k);
          __syncwarp();
        }
      }
    }
  }
}

// Links every point of the position forest straight to its root; with roots, as the
// last kernel, writes roots[index of node i] = the index of i's root in either forest.
//
// A thread moves all of its nodes up by one link a round, until none moves: every
// link's reach doubles from round to round, whatever the depth.  (A thread that
// walked one node to its root at a time walked link by link over the nodes of threads
// yet to come: 2M points along a line, numbered against the cell order, took 0.84 s,
// and a chain longer than SPIN_LIMIT failed; 215 us so.)
__global__ void __launch_bounds__(CL_THREADS) k_cluster_flatten(Control *ctl, const float4 *pts,
                                                                uint64_t *link, uint32_t *roots) {
  if (ld_relaxed_u32(&ctl->status)) return;
  const uint32_t n = uint32_t(ctl->n_points);
  const uint32_t first = blockIdx.x * CL_THREADS + threadIdx.x, step = gridDim.x * CL_THREADS;
  if (!cluster_dense(ctl)) {
    if (!roots) return;
    uint32_t *parent = reinterpret_cast<uint32_t *>(link);
    for (uint32_t i = first; i < n; i += step) roots[i] = uf_find(parent, i, &ctl->status);
    return;
  }
  bool moved = true;
  for (uint32_t round = 0; moved; ++round) {
    if (round == SPIN_LIMIT) {
      atomicOr(&ctl->status, ST_TIMEOUT);
      return;
    }
    moved = false;
    for (uint32_t i = first; i < n; i += step) {
      const uint64_t w = ld_relaxed(link + i);
      const uint64_t up = ld_relaxed(link + uint32_t(w));
      if (up == w) continue;
      st_relaxed(link + i, up);
      moved = true;
    }
  }
  if (!roots) return;
  for (uint32_t i = first; i < n; i += step) {
    const uint32_t index = __float_as_uint(pts[i].w);
    if (index < n) roots[index] = uint32_t(ld_relaxed(link + i) >> 32);
    else atomicOr(&ctl->status, ST_INTERNAL);  // cannot happen: records carry indices < n
  }
}

}  // namespace srcu
