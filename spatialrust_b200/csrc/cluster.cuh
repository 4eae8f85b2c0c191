// cluster.cuh -- Euclidean cluster roots on the radius grid.
//
// The component structure of "dx*dx + dy*dy + dz*dz <= tol*tol" (f32, the
// predicate of uniform_grid.rs:440-520 and kdtree.rs:544-549) is unique, and
// so is the reference's answer for each point: the smallest point index of
// its component (union_min_root, uniform_grid.rs:410-418; compress_roots,
// :389-395).  Here the grid of the normal estimator (cell sort, cell table,
// column hash, 3x3 column ranges) supplies the candidates, and a lock-free
// union-find links the pairs.
//
// The forest lives in cell-sorted order: the node of sorted position i is the
// word link[i] = (index of its parent point << 32) | position of its parent,
// so a warp's neighbours share sectors, where a forest over point indices
// costs a sector of its own for every neighbour.  The index in the high half
// orders the roots: a root only ever hooks under one of smaller index, by
// compare-and-swap on its own word, so every tree's root is its smallest
// member and the word of a root already is the answer.
#pragma once

#include "normals.cuh"

namespace srcu {

constexpr int CL_THREADS = 256;

__device__ __forceinline__ uint64_t uf_word(uint32_t index, uint32_t pos) {
  return (uint64_t(index) << 32) | pos;
}

// Every point a tree of its own.
__global__ void __launch_bounds__(CL_THREADS) k_cluster_init(Control *ctl, const float4 *pts,
                                                             uint64_t *link) {
  if (ld_relaxed_u32(&ctl->status)) return;
  const uint32_t n = uint32_t(ctl->n_points);
  for (uint32_t i = blockIdx.x * CL_THREADS + threadIdx.x; i < n; i += gridDim.x * CL_THREADS)
    link[i] = uf_word(__float_as_uint(pts[i].w), i);
}

// Root of node `from`, whose link was w, with path halving.  Links only ever
// move to ancestors, so the halving writes race benignly with other walks and
// with the hooks (a hook only rewrites the word of a root, which this never
// writes).
__device__ __forceinline__ uint64_t uf_find(uint64_t *link, uint32_t from, uint64_t w,
                                            uint32_t *status) {
  for (uint32_t it = 0; it < SPIN_LIMIT; ++it) {
    const uint32_t pos = uint32_t(w);
    const uint64_t up = ld_relaxed(link + pos);
    if (up == w) return w;
    if (pos != from) st_relaxed(link + from, up);
    from = pos;
    w = up;
  }
  atomicOr(status, ST_TIMEOUT);
  return w;
}

// Joins the trees of nodes i and j, whose links were a and b, and returns the
// common ancestor found.  Always the larger word climbs (Rem's algorithm:
// words fall along every path), and a root that is the larger hooks under the
// other by compare-and-swap, root or not; a swap that fails returns the link
// to climb instead.  So the smaller root -- the one nearly every join meets
// once a component has formed -- is never loaded.
__device__ __forceinline__ uint64_t uf_join(uint64_t *link, uint32_t i, uint64_t a, uint32_t j,
                                            uint64_t b, uint32_t *status) {
  for (uint32_t it = 0; it < SPIN_LIMIT; ++it) {
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
  atomicOr(status, ST_TIMEOUT);
  return b;
}

// Links every point straight to its root.
__global__ void __launch_bounds__(CL_THREADS) k_cluster_flatten(Control *ctl, uint64_t *link) {
  if (ld_relaxed_u32(&ctl->status)) return;
  const uint32_t n = uint32_t(ctl->n_points);
  for (uint32_t i = blockIdx.x * CL_THREADS + threadIdx.x; i < n; i += gridDim.x * CL_THREADS) {
    const uint64_t w = ld_relaxed(link + i);
    const uint64_t root = uf_find(link, i, w, &ctl->status);
    if (root != w) st_relaxed(link + i, root);
  }
}

// One lane per cell-sorted point i: the candidates j > i of its 27-cell
// neighbourhood (each unordered pair once) that pass the predicate are joined
// with it -- all of them, or with Sample only the first of each column.  The
// columns before the query's own in key order hold no position above i, so
// the walk starts at its own column (range 4).
//
// A lane whose point and candidate hang under different words climbs by
// dependent loads from L2 while its warp waits, so the cost is the number of
// such pairs, not the walk.  The sampled pass joins most points of a component
// through at most five pairs each; after k_cluster_flatten nearly every pair
// of the full pass hangs under one root and costs one load and a comparison.
// On the 2M-point scan at tolerance 0.3: sampled pass 206 us, flatten 52 us,
// full pass 105 us, against 690 us for the full pass alone (and 1290 us with
// both roots looked up for every pair, over point indices).
template <bool Sample>
__global__ void __launch_bounds__(CL_THREADS) k_cluster_union(Control *ctl, const float4 *pts,
                                                              const uint32_t *pt_cell,
                                                              const uint2 *ranges, float r2,
                                                              uint64_t *link) {
  if (ld_relaxed_u32(&ctl->status)) return;
  const uint32_t n = uint32_t(ctl->n_points);
  const uint64_t u_count = ctl->n_cells;
  for (uint32_t i = blockIdx.x * CL_THREADS + threadIdx.x; i < n; i += gridDim.x * CL_THREADS) {
    const float4 q = pts[i];
    const uint32_t u = pt_cell[i];
    if (u >= u_count) {  // cannot happen for a consistent cell table
      atomicOr(&ctl->status, ST_INTERNAL);
      continue;
    }
    const uint2 *rg = ranges + size_t(u) * 9;
    uint64_t root = ld_relaxed(link + i);  // the highest ancestor of i met so far
#pragma unroll 1
    for (int r = 4; r < 9; ++r) {
      const uint2 range = rg[r];
      for (uint32_t j = range.x > i + 1 ? range.x : i + 1; j < range.y; ++j) {
        const float4 c = __ldg(pts + j);
        const float dx = __fsub_rn(c.x, q.x);
        const float dy = __fsub_rn(c.y, q.y);
        const float dz = __fsub_rn(c.z, q.z);
        const float d2 =
            __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
        if (!(d2 <= r2)) continue;
        const uint64_t w = ld_relaxed(link + j);
        if (w != root) root = uf_join(link, i, root, j, w, &ctl->status);
        if (Sample) break;
      }
    }
  }
}

// roots[index of node i] = the index of i's root.
__global__ void k_cluster_roots(Control *ctl, const float4 *pts, uint64_t *link, uint32_t *roots) {
  if (ld_relaxed_u32(&ctl->status)) return;
  const uint64_t n = ctl->n_points;
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n;
       i += uint64_t(gridDim.x) * blockDim.x) {
    const uint32_t index = __float_as_uint(pts[i].w);
    const uint64_t w = uf_find(link, uint32_t(i), ld_relaxed(link + i), &ctl->status);
    if (index < n) roots[index] = uint32_t(w >> 32);
    else atomicOr(&ctl->status, ST_INTERNAL);  // cannot happen: records carry indices < n
  }
}

}  // namespace srcu
