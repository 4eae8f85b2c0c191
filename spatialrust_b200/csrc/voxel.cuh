// voxel.cuh -- bounds, voxel-key plan, and the fused segment + centroid
// reduction of the VoxelGrid centroid downsample.
#pragma once

#include "radix.cuh"

namespace srcu {

constexpr int BND_THREADS = 256;

// k_begin: zeroes the control block for a new chain, advances the epoch and
// resets the per-cloud bounds.  For a single cloud it also writes the batch
// arrays (offsets {0, n} and the cloud's parameters) so that no host copy is
// needed.
__global__ void k_begin(Control *ctl, unsigned long long n_points, Batch bt, uint32_t cloud_bits,
                        int single, VoxelParamsDev vp0, NormalParamsDev np0) {
  const uint32_t t = threadIdx.x;
  if (single && t == 0) {
    uint32_t *off = const_cast<uint32_t *>(bt.offsets);
    off[0] = 0;
    off[1] = uint32_t(n_points);
    if (bt.vparams) *const_cast<VoxelParamsDev *>(bt.vparams) = vp0;
    if (bt.nparams) *const_cast<NormalParamsDev *>(bt.nparams) = np0;
  }
  uint32_t *w = reinterpret_cast<uint32_t *>(ctl);
  const uint32_t words = sizeof(Control) / 4;
  // word 0 is the epoch
  for (uint32_t i = 1 + t; i < words; i += blockDim.x) w[i] = 0;
  for (uint32_t b = t; b < bt.clouds; b += blockDim.x) {
    Bounds z;
    for (int a = 0; a < 3; ++a) {
      z.mn[a] = 0xffffffffu;  // atomicMin target
      z.mx[a] = 0u;
    }
    z.flags = 0;
    z.pad = 0;
    bt.bounds[b] = z;
  }
  __syncthreads();
  if (t == 0) {
    ctl->epoch += EPOCHS_PER_RUN;
    ctl->n_points = n_points;
    ctl->clouds = bt.clouds;
    ctl->cloud_bits = cloud_bits;
  }
}

struct BoundsAcc {
  uint32_t mn[3], mx[3], flags;
  __device__ __forceinline__ void reset() {
    for (int a = 0; a < 3; ++a) {
      mn[a] = 0xffffffffu;
      mx[a] = 0u;
    }
    flags = 0;
  }
  __device__ __forceinline__ void add(float x, float y, float z) {
    const float v[3] = {x, y, z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      if (isnan(v[a])) {
        flags |= 1u << a;
      } else if (isinf(v[a])) {
        flags |= 8u << a;
      } else {
        const uint32_t o = f2ord(v[a]);
        mn[a] = min(mn[a], o);
        mx[a] = max(mx[a], o);
      }
    }
  }
  __device__ __forceinline__ void flush(Bounds &b) const {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      if (mn[a] != 0xffffffffu) atomicMin(&b.mn[a], mn[a]);
      if (mx[a] != 0u) atomicMax(&b.mx[a], mx[a]);
    }
    if (flags) atomicOr(&b.flags, flags);
  }
};

constexpr uint32_t BND_CHUNK = 32;  // points per lane of a warp span in the multi-cloud case

// Interleaved input records (srcu_cloud.stride > 1) -> packed columns.
struct Interleaved {
  const float *src[MAX_COLS];
  float *dst[MAX_COLS];
  uint32_t nc, stride;
};

__global__ void k_deinterleave(Interleaved iv, uint64_t n) {
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n;
       i += uint64_t(gridDim.x) * blockDim.x)
    for (uint32_t c = 0; c < iv.nc; ++c) iv.dst[c][i] = iv.src[c][i * iv.stride];
}

// k_bounds over one cloud of n points.
__device__ __forceinline__ void bounds_one_cloud(const float *x, const float *y, const float *z,
                                                 uint64_t n, const float *a0, float4 *aos,
                                                 Bounds *bounds) {
  BoundsAcc acc;
  acc.reset();
  const uint64_t stride = uint64_t(gridDim.x) * BND_THREADS;
  uint64_t i = blockIdx.x * uint64_t(BND_THREADS) + threadIdx.x;
  // four points per thread in flight: all loads first, then the stores
  for (; i + 3 * stride < n; i += 4 * stride) {
    float px[4], py[4], pz[4], pa[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint64_t k = i + uint64_t(q) * stride;
      px[q] = x[k];
      py[q] = y[k];
      pz[q] = z[k];
      pa[q] = a0 ? a0[k] : 0.0f;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (aos) aos[i + uint64_t(q) * stride] = make_float4(px[q], py[q], pz[q], pa[q]);
      acc.add(px[q], py[q], pz[q]);
    }
  }
  for (; i < n; i += stride) {
    const float xi = x[i], yi = y[i], zi = z[i];
    if (aos) aos[i] = make_float4(xi, yi, zi, a0 ? a0[i] : 0.0f);
    acc.add(xi, yi, zi);
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      acc.mn[a] = min(acc.mn[a], __shfl_xor_sync(FULL_MASK, acc.mn[a], o));
      acc.mx[a] = max(acc.mx[a], __shfl_xor_sync(FULL_MASK, acc.mx[a], o));
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc.flags |= __shfl_xor_sync(FULL_MASK, acc.flags, o);
  // one flush per block: warp results meet in shared memory first
  __shared__ uint32_t sred[BND_THREADS / 32][7];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  if (lane == 0) {
    for (int a = 0; a < 3; ++a) {
      sred[warp][a] = acc.mn[a];
      sred[warp][3 + a] = acc.mx[a];
    }
    sred[warp][6] = acc.flags;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (uint32_t w = 1; w < BND_THREADS / 32; ++w) {
      for (int a = 0; a < 3; ++a) {
        acc.mn[a] = min(acc.mn[a], sred[w][a]);
        acc.mx[a] = max(acc.mx[a], sred[w][3 + a]);
      }
      acc.flags |= sred[w][6];
    }
    acc.flush(bounds[0]);
  }
}

// k_bounds over the concatenated clouds of a batch.
__device__ __forceinline__ void bounds_many_clouds(const float *x, const float *y, const float *z,
                                                   uint64_t n, const float *a0, float4 *aos,
                                                   const Batch &bt) {
  // Many clouds: each warp owns a span of 32 * BND_CHUNK consecutive points,
  // read coalesced.  A span inside one cloud (all but at most one span per
  // cloud boundary) reduces across the warp and flushes once; a span that
  // crosses a boundary flushes per lane whenever its cloud changes.
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t span = 32ull * BND_CHUNK;
  const uint64_t spans = (n + span - 1) / span;
  const uint64_t warps = uint64_t(gridDim.x) * (BND_THREADS / 32);
  for (uint64_t sp = blockIdx.x * uint64_t(BND_THREADS / 32) + (threadIdx.x >> 5); sp < spans;
       sp += warps) {
    const uint64_t s0 = sp * span;
    const uint64_t s1 = s0 + span < n ? s0 + span : n;
    const uint32_t b0 = cloud_of(bt, uint32_t(s0));
    const uint32_t b1 = cloud_of(bt, uint32_t(s1 - 1));
    BoundsAcc acc;
    acc.reset();
    if (b0 == b1) {
      uint64_t i = s0 + lane;
      // four points per lane in flight: all loads first, then the stores
      for (; i + 96 < s1; i += 128) {
        float px[4], py[4], pz[4], pa[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint64_t k = i + 32u * q;
          px[q] = x[k];
          py[q] = y[k];
          pz[q] = z[k];
          pa[q] = a0 ? a0[k] : 0.0f;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (aos) aos[i + 32u * q] = make_float4(px[q], py[q], pz[q], pa[q]);
          acc.add(px[q], py[q], pz[q]);
        }
      }
      for (; i < s1; i += 32) {
        const float xi = x[i], yi = y[i], zi = z[i];
        if (aos) aos[i] = make_float4(xi, yi, zi, a0 ? a0[i] : 0.0f);
        acc.add(xi, yi, zi);
      }
#pragma unroll
      for (int a = 0; a < 3; ++a) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          acc.mn[a] = min(acc.mn[a], __shfl_xor_sync(FULL_MASK, acc.mn[a], o));
          acc.mx[a] = max(acc.mx[a], __shfl_xor_sync(FULL_MASK, acc.mx[a], o));
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc.flags |= __shfl_xor_sync(FULL_MASK, acc.flags, o);
      if (lane == 0) acc.flush(bt.bounds[b0]);
    } else {
      uint32_t b = b0;
      uint32_t next = __ldg(bt.offsets + b + 1);
      for (uint64_t i = s0 + lane; i < s1; i += 32) {
        while (i >= next) {  // crossed into a later cloud (skipping empty ones)
          acc.flush(bt.bounds[b]);
          acc.reset();
          ++b;
          next = __ldg(bt.offsets + b + 1);
        }
        const float xi = x[i], yi = y[i], zi = z[i];
        if (aos) aos[i] = make_float4(xi, yi, zi, a0 ? a0[i] : 0.0f);
        acc.add(xi, yi, zi);
      }
      acc.flush(bt.bounds[b]);
    }
  }
}

// Per-cloud min/max over finite coordinates plus NaN / inf flags
// (compute_bounds, voxel.rs:1067-1079, ignores NaN through f32::min/max).
// The point count comes from *count_dev when non-null, else ctl->n_points.
// Optionally writes an AoS copy (x, y, z, first attribute) so that later
// gathers by point index touch one 32-byte sector per point.
//
// The block that finishes last derives the chain's plans from the bounds: they
// move no data, so as launches of their own (voxel plans, cell plans, column
// bases) they cost a launch latency each, 10 us of a chain, against 4 us in this
// kernel's tail.  With more than PLAN_TAIL_CLOUDS clouds k_plans makes them.  Six blocks per SM: the plans' registers would leave five, which
// cost the loop 8 us at 2M points.
__global__ void __launch_bounds__(BND_THREADS, 6) k_bounds(const float *x, const float *y,
                                                        const float *z, Control *ctl,
                                                        const unsigned long long *count_dev,
                                                        const float *a0, float4 *aos, Batch bt,
                                                        PlanTasks tasks) {
  if (ld_relaxed_u32(&ctl->status)) return;
  const uint64_t n = count_dev ? *count_dev : ctl->n_points;
  if (bt.clouds == 1) bounds_one_cloud(x, y, z, n, a0, aos, bt.bounds);
  else bounds_many_clouds(x, y, z, n, a0, aos, bt);
  if (bt.clouds > PLAN_TAIL_CLOUDS) return;

  __shared__ uint32_t last;
  __shared__ unsigned long long scratch[256];
  __threadfence();  // this thread's bounds, before the block counts as done
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&ctl->work[WK_BOUNDS], 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  // the two kinds of plan do not depend on each other: half a block each
  constexpr uint32_t HALF = BND_THREADS / 2;
  const uint32_t t = threadIdx.x;
  if (tasks.voxel && t < HALF)
    for (uint32_t b = t; b < bt.clouds; b += HALF) voxel_plan(ctl, bt, b);
  if (tasks.cell && t >= HALF)
    for (uint32_t b = t - HALF; b < bt.clouds; b += HALF) cell_plan(ctl, bt, b);
  __syncthreads();
  if (tasks.cell) column_bases(ctl, bt, tasks.col_capacity, scratch);
}

// The plans of many clouds: PLAN_CLOUDS of each kind a block, and the column bases by
// the block that finishes last.
constexpr uint32_t PLAN_CLOUDS = 128;
__global__ void __launch_bounds__(2 * PLAN_CLOUDS) k_plans(Control *ctl, Batch bt, PlanTasks tasks) {
  if (ld_relaxed_u32(&ctl->status)) return;
  const uint32_t t = threadIdx.x;
  const uint32_t b = blockIdx.x * PLAN_CLOUDS + t % PLAN_CLOUDS;
  if (b < bt.clouds) {
    if (tasks.voxel && t < PLAN_CLOUDS) voxel_plan(ctl, bt, b);
    if (tasks.cell && t >= PLAN_CLOUDS) cell_plan(ctl, bt, b);
  }
  if (!tasks.cell) return;
  __shared__ uint32_t last;
  __shared__ unsigned long long scratch[256];
  __threadfence();  // this thread's plan, before the block counts as done
  __syncthreads();
  if (t == 0) last = atomicAdd(&ctl->work[WK_PLANS], 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  static_assert(2 * PLAN_CLOUDS == 256, "column_bases takes 256 threads");
  column_bases(ctl, bt, tasks.col_capacity, scratch);
}

// Key source for the voxel sort: the reference's voxel key of point i,
// packed, with its cloud id above the per-cloud key bits.
struct VoxelKeySrc {
  const float *x, *y, *z;
  Batch bt;
  VoxelPlan pl;  // the plan when there is one cloud
  uint32_t local_bits;
  uint32_t cloud_bits;
  uint32_t cloud;  // of the last key
  __device__ __forceinline__ void prepare(const Control *ctl) {
    cloud = 0;
    local_bits = ctl->vkey_bits;
    cloud_bits = ctl->cloud_bits;
    if (bt.clouds == 1) pl = bt.vplans[0];
  }
  __device__ __forceinline__ uint32_t count(const Control *ctl) const {
    return uint32_t(ctl->n_points);
  }
  __device__ __forceinline__ uint32_t key_bits() const { return local_bits + cloud_bits; }
  __device__ __forceinline__ uint64_t key(uint32_t i) {
    if (bt.clouds == 1) return voxel_pack(pl, x[i], y[i], z[i]);
    // a thread's points come in ascending order, mostly of the cloud of the last one
    // (14.6M points of 64 clouds, searched for each: 955 us for the sort, 939 so)
    if (i < __ldg(bt.offsets + cloud) || i >= __ldg(bt.offsets + cloud + 1)) cloud = cloud_of(bt, i);
    return with_cloud(voxel_pack(bt.vplans[cloud], x[i], y[i], z[i]), cloud, local_bits);
  }
};

template <int NC>
struct Columns {
  const float *in[NC];
  float *out[NC];
};

constexpr int SEG_THREADS = 256;
constexpr int SEG_ITEMS = 4;
constexpr int SEG_TILE = SEG_THREADS * SEG_ITEMS;  // 1024 sorted positions per tile
constexpr uint32_t SEG_SHORT = 32;  // longer voxels are reduced by a whole warp
constexpr int SEG_GROUP = 4;  // columns gathered and summed together
// A claimed tile keeps all later ones waiting in their look-back until it is counted, so a
// block that long voxels will hold -- the tile's average SEG_MEAN points and more, or its
// last goes on for SEG_RUN beyond it -- claims its next tile after them (2M points in
// 100 voxels: 0.82 ms with the claim ahead of them, 0.32 so; 4M in 16 53 ms and 3.6).
constexpr uint32_t SEG_MEAN = 64, SEG_RUN = 256;
// A long voxel's columns go to warps LONG_FIRST columns, then LONG_NEXT at a time; a lane
// has LONG_LOADS gathers in flight, or four items' keys.
constexpr int LONG_FIRST = 4, LONG_NEXT = 2, LONG_LOADS = 16;
constexpr int LONG_KEYS = 4;

// Shared memory of k_voxel_segments<NC>: the tile's keys (plus one before and
// one after), the scan scratch, and the tile's gathered point columns.
struct SegmentSmemHead {
  uint64_t keys[SEG_TILE + 2];  // keys[0] = key before the tile, keys[1 + tile_n] = key after it
  uint16_t start[SEG_TILE + 2];  // first position of each voxel that starts in the tile, then tile_n
  uint16_t longs[SEG_TILE / SEG_SHORT + 2];  // the tile's voxels that a warp reduces
  uint32_t ends[SEG_TILE / SEG_SHORT + 2];   // where they end among the sorted items
  uint32_t scratch[SEG_THREADS / 32];
  double inv[SEG_SHORT + 1];  // 1.0 / count of the short voxels
  uint32_t tile;              // the tile at work, then the next one
  uint32_t seg_base;
  uint32_t num_longs;
  uint32_t late;              // 1: the next tile is claimed after the long voxels
  uint64_t ahead;             // the key SEG_RUN items after the tile
};
__host__ __device__ constexpr size_t segment_smem_bytes(int nc) {
  return sizeof(SegmentSmemHead) + size_t(nc) * SEG_TILE * sizeof(float);
}

// Aggregation of the voxel whose packed key is `key`: agg_all when the host
// knows every cloud of the chain shares one, else the voxel's cloud's mode.
__device__ __forceinline__ int32_t voxel_agg(const Batch &bt, uint64_t key, uint32_t vkey_bits,
                                             int32_t agg_all) {
  if (agg_all >= 0) return agg_all;
  const uint32_t b = (bt.clouds == 1 || vkey_bits >= 64) ? 0u : uint32_t(key >> vkey_bits);
  return bt.vparams[b < bt.clouds ? b : 0].agg;
}

// Where k_voxel_segments writes a voxel besides its columns.
struct VoxelDst {
  uint64_t *keys;
  uint32_t *counts;
  float4 *aos;       // may be null
  uint32_t *starts;  // each voxel's first sorted position; may be null
  uint32_t n;
  uint32_t *status;
};

// Writes columns C0 .. C0 + G - 1 of one voxel, and with column 0 its key, count and
// AoS record.  s: their FP64 sums in ascending point order; inv: 1.0 / cnt; pos: its
// first sorted position; first(c): column c of
// the voxel's first point, read only by the modes that use it (so the default
// mode keeps no extra registers live).
//   AGG_FAST            (sum * (1.0 / count)) as f32, voxel.rs:531-536
//   AGG_CENTROID_FIRST  positions (sum / count) as f32 (average_field,
//                       voxel.rs:1156-1165), other fields from the first point
//   AGG_FIRST           every field from the first point (voxel.rs:1144-1146)
template <int NC, int C0, int G, class First>
__device__ __forceinline__ void write_centroid(const Columns<NC> &cols, const double (&s)[G],
                                               First first, int32_t agg, double inv,
                                               uint32_t pos, uint32_t cnt, uint32_t seg,
                                               uint64_t key, const VoxelDst &dst) {
  if (seg >= dst.n) {  // cannot happen for a consistent sort; never write out of bounds
    atomicOr(dst.status, ST_INTERNAL);
    return;
  }
  float o[G];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    const int c = C0 + g;
    if (agg == AGG_FAST) o[g] = __double2float_rn(__dmul_rn(s[g], inv));
    else if (agg == AGG_CENTROID_FIRST && c < 3)
      o[g] = __double2float_rn(__ddiv_rn(s[g], double(cnt)));
    else o[g] = first(c);
    cols.out[c][seg] = o[g];
  }
  if (C0 > 0) return;
  if (dst.aos) dst.aos[seg] = make_float4(o[0], o[1], o[2], 0.0f);
  if (dst.starts) dst.starts[seg] = pos;
  dst.keys[seg] = key;
  dst.counts[seg] = cnt;
}

// Columns 0 .. 3 of the points iv[]: from the AoS copy, one sector per point, where
// there is one.
template <int NC>
__device__ __forceinline__ void gather_points(float4 (&pt)[SEG_ITEMS], const uint32_t (&iv)[SEG_ITEMS],
                                              const Columns<NC> &cols, const float4 *aos_in,
                                              uint32_t n) {
#pragma unroll
  for (int q = 0; q < SEG_ITEMS; ++q) {
    pt[q] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (iv[q] >= n) continue;
    if (aos_in) {
      pt[q] = aos_in[iv[q]];
    } else {
      pt[q].x = cols.in[0][iv[q]];
      pt[q].y = cols.in[1][iv[q]];
      pt[q].z = cols.in[2][iv[q]];
      if constexpr (NC > 3) pt[q].w = cols.in[3][iv[q]];
    }
  }
}
template <int NC>
__device__ __forceinline__ void store_points(const float4 (&pt)[SEG_ITEMS], float *scol,
                                             uint32_t tile_n) {
#pragma unroll
  for (int q = 0; q < SEG_ITEMS; ++q) {
    const uint32_t j = threadIdx.x + uint32_t(q) * SEG_THREADS;
    if (j >= tile_n) continue;
    scol[0 * SEG_TILE + j] = pt[q].x;
    scol[1 * SEG_TILE + j] = pt[q].y;
    scol[2 * SEG_TILE + j] = pt[q].z;
    if constexpr (NC > 3) scol[3 * SEG_TILE + j] = pt[q].w;
  }
}
// The columns from C0 on, SEG_GROUP at a time.
template <int NC, int C0>
__device__ __forceinline__ void gather_more(const uint32_t (&iv)[SEG_ITEMS], const Columns<NC> &cols,
                                            float *scol, uint32_t tile_n, uint32_t n) {
  if constexpr (C0 < NC) {
    constexpr int G = NC - C0 < SEG_GROUP ? NC - C0 : SEG_GROUP;
    float a[SEG_ITEMS][G];
#pragma unroll
    for (int q = 0; q < SEG_ITEMS; ++q)
#pragma unroll
      for (int g = 0; g < G; ++g) a[q][g] = iv[q] < n ? cols.in[C0 + g][iv[q]] : 0.0f;
#pragma unroll
    for (int q = 0; q < SEG_ITEMS; ++q) {
      const uint32_t j = threadIdx.x + uint32_t(q) * SEG_THREADS;
      if (j >= tile_n) continue;
#pragma unroll
      for (int g = 0; g < G; ++g) scol[(C0 + g) * SEG_TILE + j] = a[q][g];
    }
    gather_more<NC, C0 + SEG_GROUP>(iv, cols, scol, tile_n, n);
  }
}

// Columns from C0 on, SEG_GROUP at a time, of the short voxel at tile positions [j, e):
// sums in ascending point index.
template <int NC, int C0>
__device__ __forceinline__ void short_voxel(const SegmentSmemHead &sm, const float *scol,
                                            uint32_t base, uint32_t j, uint32_t e, uint32_t seg,
                                            uint64_t key, const Columns<NC> &cols, int32_t agg,
                                            const VoxelDst &dst) {
  constexpr int G = NC - C0 < SEG_GROUP ? NC - C0 : SEG_GROUP;
  double s[G];
#pragma unroll
  for (int g = 0; g < G; ++g) s[g] = 0.0;
#pragma unroll 2
  for (uint32_t m = j; m < e; ++m) {
#pragma unroll
    for (int g = 0; g < G; ++g) s[g] += double(scol[(C0 + g) * SEG_TILE + m]);
  }
  write_centroid<NC, C0, G>(cols, s, [&](int c) { return scol[c * SEG_TILE + j]; }, agg,
                            sm.inv[e - j], base + j, e - j, seg, key, dst);
  if constexpr (C0 + SEG_GROUP < NC)
    short_voxel<NC, C0 + SEG_GROUP>(sm, scol, base, j, e, seg, key, cols, agg, dst);
}

// Some columns of one voxel from C0 on, its sorted items [p, e) reduced by a warp: lane l
// sums items l, l + 32, ... in order.
template <int NC, int C0>
__device__ __forceinline__ void long_voxel(const SortedView &sv, uint32_t p, uint32_t e, uint32_t seg,
                                           uint64_t key, const Columns<NC> &cols,
                                           const float4 *aos_in, int32_t agg, const VoxelDst &dst) {
  constexpr int W = C0 == 0 ? LONG_FIRST : LONG_NEXT;
  constexpr int G = NC - C0 < W ? NC - C0 : W;
  constexpr int AHEAD = LONG_LOADS / W;
  const uint32_t n = dst.n;
  const uint32_t lane = threadIdx.x & 31u;
  double s[G];
#pragma unroll
  for (int g = 0; g < G; ++g) s[g] = 0.0;
  for (uint32_t m = p + lane; m < e; m += 32 * AHEAD) {
    uint32_t v[AHEAD];
    float a[AHEAD][W];
#pragma unroll
    for (int q = 0; q < AHEAD; ++q) v[q] = m + 32 * q < e ? sv.val(m + 32 * q) : n;
    bool gathered = false;
    if constexpr (C0 == 0) {
      if (aos_in) {  // one sector per point
        gathered = true;
#pragma unroll
        for (int q = 0; q < AHEAD; ++q) {
          const float4 pt = v[q] < n ? aos_in[v[q]] : make_float4(0.f, 0.f, 0.f, 0.f);
          a[q][0] = pt.x, a[q][1] = pt.y, a[q][2] = pt.z, a[q][3] = pt.w;
        }
      }
    }
    if (!gathered) {
#pragma unroll
      for (int q = 0; q < AHEAD; ++q)
#pragma unroll
        for (int g = 0; g < G; ++g) a[q][g] = v[q] < n ? cols.in[C0 + g][v[q]] : 0.0f;
    }
#pragma unroll
    for (int q = 0; q < AHEAD; ++q) {
      if (v[q] < n) {
#pragma unroll
        for (int g = 0; g < G; ++g) s[g] += double(a[q][g]);
      } else if (m + 32 * q < e) {
        atomicOr(dst.status, ST_INTERNAL);
      }
    }
  }
#pragma unroll
  for (int g = 0; g < G; ++g)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s[g] += __shfl_xor_sync(FULL_MASK, s[g], o);
  if (lane == 0) {
    // the voxel's first point is the first sorted item (stable sort)
    auto first = [&](int c) {
      const uint32_t v0 = sv.val(p);
      return v0 < n ? cols.in[c][v0] : 0.0f;
    };
    write_centroid<NC, C0, G>(cols, s, first, agg, 1.0 / double(e - p), p, e - p, seg, key, dst);
  }
}

// The task-th share of a long voxel's columns.
template <int NC, int C0 = 0>
__device__ __forceinline__ void long_share(uint32_t task, const SortedView &sv, uint32_t p,
                                           uint32_t e, uint32_t seg, uint64_t key,
                                           const Columns<NC> &cols, const float4 *aos_in,
                                           int32_t agg, const VoxelDst &dst) {
  constexpr int NEXT = C0 + (C0 == 0 ? LONG_FIRST : LONG_NEXT);
  if (task == 0) long_voxel<NC, C0>(sv, p, e, seg, key, cols, aos_in, agg, dst);
  else if constexpr (NEXT < NC)
    long_share<NC, NEXT>(task - 1, sv, p, e, seg, key, cols, aos_in, agg, dst);
}

// Where the voxel of `key` ends, from sorted item e on, by a warp.
__device__ __forceinline__ uint32_t voxel_end(const SortedView &sv, uint64_t key, uint32_t e,
                                              uint32_t n) {
  const uint32_t lane = threadIdx.x & 31u;
  for (bool open = true; open && e < n;) {
    uint64_t at[LONG_KEYS];
#pragma unroll
    for (int k = 0; k < LONG_KEYS; ++k) at[k] = e + 32 * k + lane < n ? sv.key(e + 32 * k + lane) : ~key;
#pragma unroll
    for (int k = 0; k < LONG_KEYS; ++k) {
      const uint32_t stop = __ballot_sync(FULL_MASK, at[k] != key);
      if (open) e += stop ? __ffs(stop) - 1 : 32;
      open = open && !stop;
    }
  }
  return e;
}

// Fused segment discovery + FP64 centroid reduction over the sorted
// (key, index) pairs.  Each tile gathers its points' columns into shared
// memory with all threads at once (independent loads, so the random gather
// overlaps), flags voxel starts, numbers them with a block scan plus
// decoupled look-back, and reduces every voxel that starts in it: one thread
// per short voxel (sequential FP64 sum in ascending point index, the
// reference's order, voxel.rs:502-520), one warp per long voxel or per voxel
// that runs past the tile end.
// Bound by latency: at 2M points, 7 columns, 16% of the issue slots and a fifth of
// L2's rate are used.  So nothing waits that need not: a thread's item loads, and
// then its gathers, are issued together and stay in flight over the look-back, the
// next tile is claimed meanwhile, a thread takes a voxel (not a range of
// positions) and four columns at a time, and 64 registers keep all of that out of
// local memory.  2M points: 4 columns 83 -> 65 us, 7 columns 158 -> 97; 14.6M
// points of a batch 486 -> 380.
template <int NC>
__global__ void __launch_bounds__(SEG_THREADS, 4) k_voxel_segments(Control *ctl, SortBuffers sort,
                                                                 const SortState *sort_state,
                                                                 Columns<NC> cols,
                                                                 uint64_t *out_keys,
                                                                 uint32_t *out_counts,
                                                                 uint64_t *lookback,
                                                                 const float4 *aos_in,
                                                                 float4 *aos_out,
                                                                 uint32_t *out_starts, Batch bt,
                                                                 int32_t agg_all) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SegmentSmemHead &sm = *reinterpret_cast<SegmentSmemHead *>(smem_raw);
  float *scol = reinterpret_cast<float *>(smem_raw + sizeof(SegmentSmemHead));  // [NC][SEG_TILE]
  if (ld_relaxed_u32(&ctl->status)) return;
  const uint32_t n = uint32_t(ctl->n_points);
  if (n == 0) return;
  const SortedView sv = sorted_view(sort, *sort_state);
  const uint32_t epoch = ctl->epoch + EP_VSEG;
  const uint32_t num_tiles = (n + SEG_TILE - 1) / SEG_TILE;
  const uint32_t t = threadIdx.x, lane = t & 31u;

  const uint32_t vkey_bits = ctl->vkey_bits;
  const VoxelDst dst = {out_keys, out_counts, aos_out, out_starts, n, &ctl->status};
  if (t == 0) sm.tile = atomicAdd(&ctl->work[WK_VSEG], 1u);
  if (t >= 32 && t <= 32 + SEG_SHORT) sm.inv[t - 32] = 1.0 / double(t - 32);

  for (;;) {
    __syncthreads();
    const uint32_t tile = sm.tile;
    if (tile >= num_tiles) break;
    const uint32_t base = tile * SEG_TILE;
    const uint32_t tile_n = min(uint32_t(SEG_TILE), n - base);
    // The tile's sorted items, then their points: every thread issues all of
    // its SEG_ITEMS item loads, then all of its random point gathers, before
    // any of them is consumed, so the gathers' latencies overlap -- with one
    // another, and with the count of the voxel starts and the look-back over it,
    // which need the keys alone.
    uint32_t iv[SEG_ITEMS];
    {
      uint64_t w[SEG_ITEMS], edge = 0;  // edge: the item either side of the tile (threads 0 and 1)
#pragma unroll
      for (int q = 0; q < SEG_ITEMS; ++q) {
        const uint32_t j = t + uint32_t(q) * SEG_THREADS;
        w[q] = j < tile_n ? sv.keys[base + j] : 0ull;
      }
      if (t == 0) edge = sv.keys[base > 0 ? base - 1 : 0u];
      if (t == 1) edge = sv.keys[base + tile_n < n ? base + tile_n : n - 1];
      if (t == 2) edge = sv.keys[base + tile_n + SEG_RUN < n ? base + tile_n + SEG_RUN : n - 1];
      if (!sv.packed) {
#pragma unroll
        for (int q = 0; q < SEG_ITEMS; ++q) {
          const uint32_t j = t + uint32_t(q) * SEG_THREADS;
          iv[q] = j < tile_n ? sv.vals[base + j] : n;  // out of range: no gather
        }
      } else {
#pragma unroll
        for (int q = 0; q < SEG_ITEMS; ++q) {
          const uint32_t j = t + uint32_t(q) * SEG_THREADS;
          iv[q] = j < tile_n ? uint32_t(w[q] & ((1ull << sv.idx_bits) - 1)) : n;
        }
      }
      const uint32_t key_shift = sv.packed ? sv.idx_bits : 0u;
#pragma unroll
      for (int q = 0; q < SEG_ITEMS; ++q) {
        const uint32_t j = t + uint32_t(q) * SEG_THREADS;
        if (j >= tile_n) continue;
        sm.keys[1 + j] = w[q] >> key_shift;
        // a consistent sort never produces this; never read out of bounds
        if (iv[q] >= n) atomicOr(&ctl->status, ST_INTERNAL);
      }
      edge >>= key_shift;
      if (t == 0) {  // unlike the first key where there is none before it
        sm.keys[0] = base > 0 ? edge : ~edge;
        sm.num_longs = 0;
      }
      if (t == 1) sm.keys[1 + tile_n] = base + tile_n < n ? edge : ~edge;
      if (t == 2) sm.ahead = base + tile_n + SEG_RUN < n ? edge : ~edge;
    }
    float4 pt[SEG_ITEMS];
    gather_points<NC>(pt, iv, cols, aos_in, n);
    __syncthreads();

    const uint32_t j0 = t * SEG_ITEMS;
    uint32_t flags = 0;
#pragma unroll
    for (int i = 0; i < SEG_ITEMS; ++i) {
      const uint32_t j = j0 + i;
      if (j < tile_n && sm.keys[1 + j] != sm.keys[j]) flags |= 1u << i;
    }
    uint32_t voxels;
    uint32_t local = block_exclusive_sum<SEG_THREADS>(__popc(flags), sm.scratch, &voxels);
    if (t < 32) {
      const uint32_t seg_base =
          lookback_exclusive_warp(lookback, tile, voxels, epoch, &ctl->status,
                                  num_tiles <= gridDim.x);
      if (t == 0) {
        sm.seg_base = seg_base;
        sm.late = voxels * SEG_MEAN < tile_n || sm.ahead == sm.keys[tile_n];
        if (!sm.late) sm.tile = atomicAdd(&ctl->work[WK_VSEG], 1u);
        sm.start[voxels] = uint16_t(tile_n);
        if (tile == num_tiles - 1) ctl->n_voxels = seg_base + voxels;
      }
    }
#pragma unroll
    for (int i = 0; i < SEG_ITEMS; ++i)
      if (flags & (1u << i)) sm.start[local++] = uint16_t(j0 + i);
    store_points<NC>(pt, scol, tile_n);
    gather_more<NC, 4>(iv, cols, scol, tile_n, n);
    __syncthreads();

    // Short voxels: a thread each, from shared memory.  Long ones (more than SEG_SHORT
    // points, or running past the tile) are listed.
    for (uint32_t q = t; q < voxels; q += SEG_THREADS) {
      const uint32_t j = sm.start[q], e = sm.start[q + 1];
      const uint64_t key = sm.keys[1 + j];
      if (e - j > SEG_SHORT || sm.keys[1 + e] == key)
        sm.longs[atomicAdd(&sm.num_longs, 1u)] = uint16_t(q);
      else
        short_voxel<NC, 0>(sm, scol, base, j, e, sm.seg_base + q, key, cols,
                           voxel_agg(bt, key, vkey_bits, agg_all), dst);
    }
    __syncthreads();
    // Long voxels: a warp finds the end; then a warp for every share of its columns reduces
    // them from global memory.  With one warp for all columns, an item at a time, and the
    // next tile claimed before, 2M points in 1600 voxels took 373 us at three columns and
    // 1934 at twelve, 119 and 457 so; in 100 voxels 2.3 and 12.7 ms, 0.32 and 0.76.
    if (const uint32_t longs = sm.num_longs) {
      for (uint32_t i = t >> 5; i < longs; i += SEG_THREADS / 32) {
        const uint32_t q = sm.longs[i];
        const uint32_t e = voxel_end(sv, sm.keys[1 + sm.start[q]], base + sm.start[q + 1], n);
        if (lane == 0) sm.ends[i] = e;
      }
      __syncthreads();
      constexpr uint32_t SHARES =
          NC <= LONG_FIRST ? 1 : 1 + (NC - LONG_FIRST + LONG_NEXT - 1) / LONG_NEXT;
      for (uint32_t i = t >> 5; i < longs * SHARES; i += SEG_THREADS / 32) {
        const uint32_t q = sm.longs[i / SHARES];
        const uint64_t key = sm.keys[1 + sm.start[q]];
        long_share<NC>(i % SHARES, sv, base + sm.start[q], sm.ends[i / SHARES], sm.seg_base + q,
                       key, cols, aos_in, voxel_agg(bt, key, vkey_bits, agg_all), dst);
      }
    }
    if (t == 0 && sm.late) sm.tile = atomicAdd(&ctl->work[WK_VSEG], 1u);
  }
}

// Opts every k_voxel_segments<NC> instantiation into the shared memory it
// needs (more than 48 KB for many attribute columns).
template <int NC>
inline cudaError_t configure_segments_nc() {
  return cudaFuncSetAttribute(k_voxel_segments<NC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              int(segment_smem_bytes(NC)));
}
inline cudaError_t configure_segment_kernels() {
  cudaError_t e = cudaSuccess;
  const cudaError_t all[] = {configure_segments_nc<3>(),  configure_segments_nc<4>(),
                             configure_segments_nc<5>(),  configure_segments_nc<6>(),
                             configure_segments_nc<7>(),  configure_segments_nc<8>(),
                             configure_segments_nc<9>(),  configure_segments_nc<10>(),
                             configure_segments_nc<11>(), configure_segments_nc<12>()};
  for (cudaError_t x : all)
    if (x != cudaSuccess) e = x;
  return e;
}

// ---- the reference's plain-xyz fast path --------------------------------------
// filter_cpu_xyz_centroid_fast (crates/spatialrust-filtering/src/voxel.rs:550-636)
// runs for clouds whose only fields are x, y, z: per voxel it sums x, y, z in
// f32 in input order, emits sum * (1 / count) in f32, and emits the voxels in
// the order of their first point.  After the segment kernel (same voxels, same
// counts, key order, and where each voxel's sorted items start), k_voxel_xyz_f32
// recomputes those sums -- the stable sort keeps each voxel's points in input
// order -- and marks each voxel's first point with the voxel; the count of marks
// before a point is then its voxel's place, so one scan over the points
// (k_voxel_first_seen) puts the voxels in first-seen order, without a sort.
// Both kernels are bound by the latency of their gathers (11 and 21 us at 300k points
// with cold caches).  With a sort of the voxels by first point (40 us alone), a
// gather, a copy back and a binary search per voxel in their place, a call from
// host memory took 663 us; it takes 612.

constexpr uint32_t XYZ_THREADS = 256;
constexpr uint32_t XYZ_SHORT = 128;  // points of a voxel that its thread sums alone

// One thread per voxel; a voxel of more than XYZ_SHORT points is summed by its warp,
// whose lanes gather 32 points at a time, the next 32 while three of them add a
// coordinate each in order (one thread alone waits for the gathers: 100 voxels of 20k
// points 27 ms, 1.7 so).  `starts` and tx may be the same memory: a
// thread reads its start before it writes.  mark: a word per point, zeroed.
__global__ void __launch_bounds__(XYZ_THREADS) k_voxel_xyz_f32(
    Control *ctl, SortBuffers sort, const SortState *sort_state, const float4 *aos,
    const uint64_t *vkeys, const uint32_t *vcounts, const uint32_t *starts, float *tx, float *ty,
    float *tz, uint32_t *tc, uint64_t *tk, uint32_t *mark) {
  __shared__ float rows[XYZ_THREADS / 32][3][32];
  if (ld_relaxed_u32(&ctl->status)) return;
  const uint32_t n = uint32_t(ctl->n_points);
  const uint32_t nv = uint32_t(ctl->n_voxels);
  const SortedView sv = sorted_view(sort, *sort_state);
  const uint32_t lane = threadIdx.x & 31u;
  float(*row)[32] = rows[threadIdx.x >> 5];
  // few voxels are spread over the warps: a warp takes its long ones one after another
  const uint32_t warps = gridDim.x * (XYZ_THREADS / 32);
  const uint32_t per = max(1u, min(32u, (nv + warps - 1) / warps));
  for (uint32_t v0 = (blockIdx.x * (XYZ_THREADS / 32) + (threadIdx.x >> 5)) * per; v0 < nv;
       v0 += warps * per) {
    const uint32_t v = v0 + lane;
    uint32_t m = 0, cnt = 0;
    uint64_t key = 0;
    bool ok = lane < per && v < nv;
    if (ok) {
      m = starts[v];
      cnt = vcounts[v];
      key = vkeys[v];
      ok = m < n && cnt > 0 && cnt <= n - m;
      if (!ok) atomicOr(&ctl->status, ST_INTERNAL);  // cannot happen for a consistent chain
    }
    auto point = [&](uint32_t at, bool in, bool &good) {
      const uint32_t i = in ? sv.val(at) : n;
      good &= !in || i < n;
      return i < n ? aos[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    float sx = 0.0f, sy = 0.0f, sz = 0.0f;
    if (ok && cnt <= XYZ_SHORT) {
#pragma unroll 4
      for (uint32_t q = 0; q < cnt; ++q) {
        const float4 p = point(m + q, true, ok);
        sx = __fadd_rn(sx, p.x);
        sy = __fadd_rn(sy, p.y);
        sz = __fadd_rn(sz, p.z);
      }
      if (!ok) atomicOr(&ctl->status, ST_INTERNAL);
    }
    for (uint32_t todo = __ballot_sync(FULL_MASK, ok && cnt > XYZ_SHORT); todo; todo &= todo - 1) {
      const uint32_t owner = __ffs(todo) - 1;
      const uint32_t m0 = __shfl_sync(FULL_MASK, m, owner), c0 = __shfl_sync(FULL_MASK, cnt, owner);
      bool good = true;
      float sum = 0.0f;  // lanes 0 to 2: x, y, z
      float4 next = point(m0 + lane, lane < c0, good);
      for (uint32_t q = 0; q < c0; q += 32) {
        row[0][lane] = next.x;
        row[1][lane] = next.y;
        row[2][lane] = next.z;
        __syncwarp();
        if (q + 32 < c0) next = point(m0 + q + 32 + lane, q + 32 + lane < c0, good);
        if (lane < 3) {
          const uint32_t k = min(32u, c0 - q);
          if (k == 32) {
#pragma unroll
            for (uint32_t j = 0; j < 32; ++j) sum = __fadd_rn(sum, row[lane][j]);
          } else {
            for (uint32_t j = 0; j < k; ++j) sum = __fadd_rn(sum, row[lane][j]);
          }
        }
        __syncwarp();
      }
      good = __all_sync(FULL_MASK, good);
      const float x = __shfl_sync(FULL_MASK, sum, 0), y = __shfl_sync(FULL_MASK, sum, 1);
      const float z = __shfl_sync(FULL_MASK, sum, 2);
      if (lane == owner) {
        sx = x, sy = y, sz = z;
        ok = good;
        if (!good) atomicOr(&ctl->status, ST_INTERNAL);
      }
    }
    if (!ok) continue;
    const float inv = 1.0f / float(cnt);  // IEEE division: the library is built without fast math
    tx[v] = __fmul_rn(sx, inv);
    ty[v] = __fmul_rn(sy, inv);
    tz[v] = __fmul_rn(sz, inv);
    tc[v] = cnt;
    tk[v] = key;
    mark[sv.val(m)] = v + 1;
  }
}

// The voxels into the chain's buffers (and the AoS copy the normals stage reads) in
// the order of their marks: a count of marks over tiles of SEG_TILE points, with a
// look-back, a thread to four consecutive points.
__global__ void __launch_bounds__(SEG_THREADS) k_voxel_first_seen(
    Control *ctl, const uint32_t *mark, uint64_t *lookback, const float *tx, const float *ty,
    const float *tz, const uint32_t *tc, const uint64_t *tk, float *ox, float *oy, float *oz,
    uint32_t *ocnt, uint64_t *okey, float4 *oaos) {
  __shared__ uint32_t scratch[SEG_THREADS / 32];
  __shared__ uint32_t s_tile, s_base;
  if (ld_relaxed_u32(&ctl->status)) return;
  const uint32_t n = uint32_t(ctl->n_points);
  const uint32_t nv = uint32_t(ctl->n_voxels);
  const uint32_t num_tiles = (n + SEG_TILE - 1) / SEG_TILE;
  const uint32_t t = threadIdx.x;
  if (t == 0) s_tile = atomicAdd(&ctl->work[WK_ORDER], 1u);
  for (;;) {
    __syncthreads();
    const uint32_t tile = s_tile;
    if (tile >= num_tiles) break;
    const uint32_t i0 = tile * SEG_TILE + t * SEG_ITEMS;
    uint32_t v[SEG_ITEMS], marks = 0;
#pragma unroll
    for (int q = 0; q < SEG_ITEMS; ++q) v[q] = i0 + q < n ? mark[i0 + q] : 0u;
#pragma unroll
    for (int q = 0; q < SEG_ITEMS; ++q) marks += v[q] != 0;
    uint32_t total;
    const uint32_t local = block_exclusive_sum<SEG_THREADS>(marks, scratch, &total);
    if (t < 32) {
      const uint32_t base = lookback_exclusive_warp(lookback, tile, total, ctl->epoch + EP_ORDER,
                                                    &ctl->status, num_tiles <= gridDim.x);
      if (t == 0) {
        s_base = base;
        s_tile = atomicAdd(&ctl->work[WK_ORDER], 1u);  // the next one
        // every voxel has marked one point
        if (tile == num_tiles - 1 && base + total != nv) atomicOr(&ctl->status, ST_INTERNAL);
      }
    }
    __syncthreads();
    uint32_t j = s_base + local;
#pragma unroll
    for (int q = 0; q < SEG_ITEMS; ++q) {
      if (v[q] == 0) continue;
      const uint32_t u = v[q] - 1;
      if (u < nv && j < nv) {
        const float x = tx[u], y = ty[u], z = tz[u];
        ox[j] = x;
        oy[j] = y;
        oz[j] = z;
        if (oaos) oaos[j] = make_float4(x, y, z, 0.0f);
        ocnt[j] = tc[u];
        okey[j] = tk[u];
      } else {
        atomicOr(&ctl->status, ST_INTERNAL);
      }
      ++j;
    }
  }
}

// Unpacks packed voxel keys into the reference's (ix, iy, iz) int64 triples.
__global__ void k_unpack_voxel_keys(const Control *ctl, const uint64_t *packed, int64_t *out,
                                    Batch bt) {
  if (ctl->status) return;
  const uint64_t v = ctl->n_voxels;
  const uint32_t lb = ctl->vkey_bits;
  const uint64_t mask = lb >= 64 ? ~0ull : ((1ull << lb) - 1);
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < v;
       i += uint64_t(gridDim.x) * blockDim.x) {
    const uint64_t key = packed[i];
    const uint32_t b = lb >= 64 ? 0u : uint32_t(key >> lb);
    int64_t k[3];
    voxel_unpack(bt.vplans[b < bt.clouds ? b : 0], key & mask, k);
    out[3 * i] = k[0];
    out[3 * i + 1] = k[1];
    out[3 * i + 2] = k[2];
  }
}

// Voxel range of every cloud in the key-ordered output: voxel_offsets[b] is
// the first voxel whose key carries cloud id >= b (binary search).
__global__ void k_voxel_offsets(const Control *ctl, const uint64_t *packed, Batch bt) {
  if (ctl->status) return;
  const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b > bt.clouds) return;
  const uint64_t v = ctl->n_voxels;
  const uint32_t lb = ctl->vkey_bits;
  uint64_t lo = 0, hi = v;
  if (b == 0) hi = 0;
  else if (b == bt.clouds) lo = v;
  else {
    const uint64_t target = uint64_t(b) << lb;  // lb < 64 whenever there are 2+ clouds
    while (lo < hi) {
      const uint64_t mid = (lo + hi) >> 1;
      if (packed[mid] < target) lo = mid + 1;
      else hi = mid;
    }
  }
  bt.voxel_offsets[b] = uint32_t(lo);
}

}  // namespace srcu
