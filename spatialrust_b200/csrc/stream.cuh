// stream.cuh -- bounded streaming voxel centroids on the device, the
// counterpart of StreamingVoxelSource
// (crates/spatialrust-pipeline/src/streaming.rs:334-700).
//
// Semantics followed (streaming.rs):
//   - the voxel of a point is floor(f64(v) / f64(leaf)) per axis, no origin
//     (voxel_coordinate, :986-994); a coordinate outside the i64 range is an
//     error;
//   - points with a non-finite coordinate are skipped (:464-466);
//   - every column of a voxel is averaged in FP64 over all its points of the
//     whole stream, sum / count (:852-858, :631-633);
//   - voxels come out in ascending (ix, iy, iz) order (:805-838).
//
// Device design.  Chunks are packed into a device run buffer, one record per
// point.  A full run is sorted by packed key with the onesweep sort (stable, so
// a voxel's points stay in stream order) and reduced to partial records -- key,
// count and a compensated FP64 sum of every column -- appended to a device
// record store.  finish() sorts all partial records by key (stable, so runs stay
// in stream order) and reduces them again, straight into the outputs; a stream
// that fits one run is reduced into the outputs at once.  Only reduced runs stay
// resident: device memory grows with the distinct voxels of each run, not with
// the length of the stream.
//
// The reductions gather points in key order, which is random in the run buffer.
// A packed record is one 32-byte sector for up to four f32 and two f64 columns,
// where the columns apart cost a sector each (run reduction of 4.2M points of
// three positions and two attributes: 580 us and 1.6 GB read; 193 us here).
//
// A voxel's sum is compensated (Kahan) within each run and across runs, as
// the reference's CompensatedSum is over the whole stream (:240-262); the
// grouping differs, so means agree to FP64 rounding, not bit for bit.
#pragma once

#include <climits>

#include "radix.cuh"

namespace srcu {

constexpr int SV_THREADS = 256;
constexpr int SV_ITEMS = 4;
constexpr int SV_TILE = SV_THREADS * SV_ITEMS;  // sorted positions per tile
constexpr uint32_t SV_SHORT = 64;  // longer segments are reduced by a whole block
// Of those: points a thread loads before it adds them.  A sum alone in its loop waits
// for each point (2M points of five columns in one voxel: 11.1 ms, 5.8 with four ahead;
// in some 800 voxels 1.03 ms, 0.70).
constexpr uint32_t SV_AHEAD = 4;
constexpr double SV_I64_EDGE = 9223372036854775808.0;  // 2^63: i64::MIN and i64::MAX as f64

// Packing of one sort: per-axis key minimum and bit widths.  Bit total_bits
// of a packed key marks a skipped (non-finite) point, which sorts last.
struct StreamPlan {
  long long kmin[3];
  uint32_t bits[3];
  uint32_t shift_y, shift_x;
  uint32_t total_bits;
  uint32_t any;  // 1: the sort holds at least one finite point
  uint32_t pad;
};

// Device state of one stream.
struct StreamState {
  long long gmin[3], gmax[3];      // key range over every run's finite points
  unsigned long long finite;       // finite points over all runs
  unsigned long long segments;     // records written by the last reduction
  unsigned long long long_count;   // long segments of the last reduction
  uint32_t overflow;               // 1: a key leaves the i64 range; 2: packed key > 63 bits
  uint32_t pad;
};

// Packed point records: the f64 columns, then the f32 columns in pairs, padded
// to 16-byte units.  The positions are the first three f32 columns.
struct StreamLayout {
  uint32_t nc, nd, nf;  // columns: all, f64, f32
  uint32_t units;       // 16-byte units per record
  uint32_t col_d[MAX_COLS], col_f[MAX_COLS];  // the column behind each f64 / f32 field
};

// One reduction's inputs: packed points, or the partial records' FP64 sums and
// counts.
struct StreamIn {
  const uint4 *points;
  StreamLayout lay;
  const double *sum[MAX_COLS];    // records only
  const unsigned long long *cnt;  // records only
};

// One reduction's outputs, written at base + slot < cap: the partial record
// store (SoA), or with Final the stream's own -- positions as f32, the other
// columns' means in FP64 (narrowed by the caller per field type, as push_scalar
// does, streaming.rs:922-938), (ix, iy, iz) triples.
struct StreamOut {
  long long *kx, *ky, *kz;
  unsigned long long *cnt;
  double *sum[MAX_COLS];
  float *pos[3];
  double *attr[MAX_COLS];
  long long *keys3;
  unsigned long long base, cap;
};

// floor(v / leaf) in FP64 as an i64 (streaming.rs:986-994): false when the
// result leaves the range; 2^63 itself saturates like Rust's `as i64`.
__device__ __forceinline__ bool stream_axis_key(float v, double leaf, long long &k) {
  const double c = floor(__ddiv_rn(double(v), leaf));
  if (c < -SV_I64_EDGE || c > SV_I64_EDGE) return false;
  k = c >= SV_I64_EDGE ? LLONG_MAX : (long long)c;
  return true;
}

__device__ __forceinline__ uint64_t stream_pack(const StreamPlan &pl, long long kx, long long ky,
                                                long long kz) {
  const uint64_t fx = uint64_t(kx) - uint64_t(pl.kmin[0]);
  const uint64_t fy = uint64_t(ky) - uint64_t(pl.kmin[1]);
  const uint64_t fz = uint64_t(kz) - uint64_t(pl.kmin[2]);
  return (fx << pl.shift_x) | (fy << pl.shift_y) | fz;
}

__device__ __forceinline__ void stream_unpack(const StreamPlan &pl, uint64_t key, long long &kx,
                                              long long &ky, long long &kz) {
  const uint64_t mz = pl.bits[2] ? (~0ull >> (64 - pl.bits[2])) : 0ull;
  const uint64_t my = pl.bits[1] ? (~0ull >> (64 - pl.bits[1])) : 0ull;
  kz = (long long)(uint64_t(pl.kmin[2]) + (key & mz));
  ky = (long long)(uint64_t(pl.kmin[1]) + ((key >> pl.shift_y) & my));
  kx = (long long)(uint64_t(pl.kmin[0]) + (pl.shift_x < 64 ? (key >> pl.shift_x) : 0ull));
}

__device__ __forceinline__ bool finite3(float x, float y, float z) {
  return isfinite(x) && isfinite(y) && isfinite(z);
}

__device__ __forceinline__ float3 stream_pos(const uint4 *points, const StreamLayout &lay,
                                             uint64_t i) {
  const float *f = reinterpret_cast<const float *>(points + i * lay.units) + 2 * lay.nd;
  return make_float3(f[0], f[1], f[2]);
}

// A chunk's columns -> packed records.
struct StreamChunk {
  const void *col[MAX_COLS];
};
__global__ void __launch_bounds__(256) k_stream_pack(const __grid_constant__ StreamChunk ch,
                                                     const __grid_constant__ StreamLayout lay,
                                                     uint64_t n, uint4 *points) {
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n;
       i += uint64_t(gridDim.x) * blockDim.x) {
    auto pair = [&](uint32_t p) -> uint2 {  // 8 bytes: one f64 field or two f32 fields
      uint2 w = make_uint2(0, 0);
      if (p < lay.nd) return static_cast<const uint2 *>(ch.col[lay.col_d[p]])[i];
      const uint32_t f = 2 * (p - lay.nd);
      if (f < lay.nf) w.x = static_cast<const uint32_t *>(ch.col[lay.col_f[f]])[i];
      if (f + 1 < lay.nf) w.y = static_cast<const uint32_t *>(ch.col[lay.col_f[f + 1]])[i];
      return w;
    };
    for (uint32_t u = 0; u < lay.units; ++u) {
      const uint2 a = pair(2 * u), b = pair(2 * u + 1);
      points[i * lay.units + u] = make_uint4(a.x, a.y, b.x, b.y);
    }
  }
}

// Per-axis min/max over the points whose three coordinates are finite (the
// points the stream keeps) of the current run (ctl->n_points of them):
// warp then block reductions, six atomics per block.
__global__ void __launch_bounds__(256) k_stream_bounds(Control *ctl, const uint4 *points,
                                                       StreamLayout lay, Bounds *out) {
  __shared__ uint32_t red[6][8];
  if (ld_relaxed_u32(&ctl->status)) return;
  const uint64_t n = ctl->n_points;
  uint32_t v6[6] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0u, 0u, 0u};  // mn xyz, mx xyz
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n;
       i += uint64_t(gridDim.x) * blockDim.x) {
    const float3 p = stream_pos(points, lay, i);
    const float v[3] = {p.x, p.y, p.z};
    if (!finite3(v[0], v[1], v[2])) continue;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const uint32_t o = f2ord(v[a]);
      v6[a] = min(v6[a], o);
      v6[3 + a] = max(v6[3 + a], o);
    }
  }
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    v6[a] = __reduce_min_sync(FULL_MASK, v6[a]);
    v6[3 + a] = __reduce_max_sync(FULL_MASK, v6[3 + a]);
  }
  if (lane == 0)
    for (int k = 0; k < 6; ++k) red[k][warp] = v6[k];
  __syncthreads();
  if (threadIdx.x == 0) {
    const uint32_t warps = blockDim.x >> 5;
    for (int a = 0; a < 3; ++a) {
      uint32_t mn = red[a][0], mx = red[3 + a][0];
      for (uint32_t w = 1; w < warps; ++w) {
        mn = min(mn, red[a][w]);
        mx = max(mx, red[3 + a][w]);
      }
      if (mn != 0xffffffffu) {
        atomicMin(&out->mn[a], mn);
        atomicMax(&out->mx[a], mx);
      }
    }
  }
}

__device__ __forceinline__ void stream_plan_finish(StreamPlan &pl, const long long (&kmax)[3],
                                                   Control *ctl, StreamState *st) {
  uint32_t total = 0;
  for (int a = 0; a < 3; ++a) {
    pl.bits[a] = bit_width_u64(uint64_t(kmax[a]) - uint64_t(pl.kmin[a]));
    total += pl.bits[a];
  }
  pl.shift_y = pl.bits[2];
  pl.shift_x = pl.bits[1] + pl.bits[2];
  pl.total_bits = total;
  if (total > 63) {
    st->overflow = 2;
    atomicOr(&ctl->status, ST_KEY_OVERFLOW);
  }
}

// Plan of one run from its bounds; widens the stream's key range.  One thread.
__global__ void k_stream_plan(Control *ctl, const Bounds *bd, double leaf, StreamPlan *plan,
                              StreamState *st) {
  if (threadIdx.x != 0 || ld_relaxed_u32(&ctl->status)) return;
  StreamPlan pl{};
  const Bounds b = *bd;
  pl.any = (b.mn[0] != 0xffffffffu) ? 1u : 0u;  // all three axes or none
  long long kmax[3] = {0, 0, 0};
  if (pl.any) {
    for (int a = 0; a < 3; ++a) {
      long long lo, hi;
      if (!stream_axis_key(ord2f(b.mn[a]), leaf, lo) || !stream_axis_key(ord2f(b.mx[a]), leaf, hi)) {
        st->overflow = 1;
        atomicOr(&ctl->status, ST_KEY_OVERFLOW);
        return;
      }
      pl.kmin[a] = lo;
      kmax[a] = hi;
      atomicMin(&st->gmin[a], lo);
      atomicMax(&st->gmax[a], hi);
    }
  }
  stream_plan_finish(pl, kmax, ctl, st);
  *plan = pl;
}

// Plan of the final merge: the key range of every run.  One thread.
__global__ void k_stream_merge_plan(Control *ctl, StreamPlan *plan, StreamState *st) {
  if (threadIdx.x != 0 || ld_relaxed_u32(&ctl->status)) return;
  StreamPlan pl{};
  long long kmax[3] = {0, 0, 0};
  pl.any = st->gmin[0] <= st->gmax[0] ? 1u : 0u;
  if (pl.any)
    for (int a = 0; a < 3; ++a) {
      pl.kmin[a] = st->gmin[a];
      kmax[a] = st->gmax[a];
    }
  stream_plan_finish(pl, kmax, ctl, st);
  *plan = pl;
}

// Sort key of a run's points (ctl->n_points of them).
struct StreamPointSrc {
  const uint4 *points;
  StreamLayout lay;
  const StreamPlan *plan_ptr;
  double leaf;
  StreamPlan pl;
  __device__ __forceinline__ void prepare(const Control *) { pl = *plan_ptr; }
  __device__ __forceinline__ uint32_t count(const Control *ctl) const { return uint32_t(ctl->n_points); }
  __device__ __forceinline__ uint32_t key_bits() const { return pl.total_bits + 1; }
  __device__ __forceinline__ uint64_t key(uint32_t i) const {
    const float3 p = stream_pos(points, lay, i);
    long long kx, ky, kz;
    // a finite point lies inside the run's bounds, so its keys are in range
    if (!finite3(p.x, p.y, p.z) || !stream_axis_key(p.x, leaf, kx) ||
        !stream_axis_key(p.y, leaf, ky) || !stream_axis_key(p.z, leaf, kz))
      return 1ull << pl.total_bits;
    return stream_pack(pl, kx, ky, kz);
  }
};

// Sort key of the partial records (ctl->n_points of them).
struct StreamRecordSrc {
  const long long *kx, *ky, *kz;
  const StreamPlan *plan_ptr;
  StreamPlan pl;
  __device__ __forceinline__ void prepare(const Control *) { pl = *plan_ptr; }
  __device__ __forceinline__ uint32_t count(const Control *ctl) const { return uint32_t(ctl->n_points); }
  __device__ __forceinline__ uint32_t key_bits() const { return pl.total_bits + 1; }
  __device__ __forceinline__ uint64_t key(uint32_t i) const {
    return stream_pack(pl, kx[i], ky[i], kz[i]);
  }
};

// A sorted position starts a voxel: kept, and first or unlike its predecessor.
__device__ __forceinline__ bool stream_head(const SortedView &sv, uint64_t flag, uint32_t i,
                                            uint64_t &key) {
  key = sv.key(i);
  if (key & flag) return false;
  return i == 0 || sv.key(i - 1) != key;
}

// Voxel starts per tile of SV_TILE sorted positions (thread t owns positions
// 4t .. 4t+3 of the tile); kept points into st->finite when count_finite.
__global__ void __launch_bounds__(SV_THREADS) k_stream_flags(Control *ctl, SortBuffers sort,
                                                             const SortState *ss,
                                                             const StreamPlan *plan,
                                                             uint32_t *tile_heads, StreamState *st,
                                                             int count_finite) {
  __shared__ uint32_t scratch[SV_THREADS / 32];
  if (ld_relaxed_u32(&ctl->status)) return;
  const uint32_t n = uint32_t(ctl->n_points);
  const uint32_t tiles = (n + SV_TILE - 1) / SV_TILE;
  const SortedView sv = sorted_view(sort, *ss);
  const uint64_t flag = 1ull << plan->total_bits;
  for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    uint32_t heads = 0, kept = 0;
#pragma unroll
    for (int k = 0; k < SV_ITEMS; ++k) {
      const uint32_t i = tile * SV_TILE + threadIdx.x * SV_ITEMS + k;
      if (i >= n) break;
      uint64_t key;
      heads += stream_head(sv, flag, i, key) ? 1u : 0u;
      kept += (key & flag) ? 0u : 1u;
    }
    uint32_t total_heads, total_kept;
    block_exclusive_sum<SV_THREADS>(heads, scratch, &total_heads);
    block_exclusive_sum<SV_THREADS>(kept, scratch, &total_kept);
    if (threadIdx.x == 0) {
      tile_heads[tile] = total_heads;
      if (count_finite && total_kept) atomicAdd(&st->finite, (unsigned long long)total_kept);
    }
  }
}

// Exclusive scan of the tile counts (one block of 1024 threads); the total
// is the number of records the reduction writes.
__global__ void __launch_bounds__(1024) k_stream_scan(Control *ctl, const uint32_t *tile_heads,
                                                      uint32_t *tile_off, StreamState *st) {
  __shared__ uint32_t scratch[32];
  if (ld_relaxed_u32(&ctl->status)) return;
  const uint32_t n = uint32_t(ctl->n_points);
  const uint32_t tiles = (n + SV_TILE - 1) / SV_TILE;
  const uint32_t per = (tiles + 1023) / 1024;
  const uint32_t lo = min(tiles, threadIdx.x * per), hi = min(tiles, lo + per);
  uint32_t local = 0;
  for (uint32_t t = lo; t < hi; ++t) local += tile_heads[t];
  uint32_t total;
  uint32_t run = block_exclusive_sum<1024>(local, scratch, &total);
  for (uint32_t t = lo; t < hi; ++t) {
    tile_off[t] = run;
    run += tile_heads[t];
  }
  if (threadIdx.x == 0) {
    st->segments = total;
    st->long_count = 0;
    ctl->n_voxels = total;
  }
}

// Compensated sum (Kahan): the running correction is subtracted from each
// addend, as CompensatedSum::add does (streaming.rs:246-257).
struct Kahan {
  double s = 0.0, c = 0.0;
  __device__ __forceinline__ void add(double v) {
    const double y = __dsub_rn(v, c);
    const double t = __dadd_rn(s, y);
    c = __dsub_rn(__dsub_rn(t, s), y);
    s = t;
  }
};

// Key and count of output record r; one column's sum, or its mean with Final.
template <bool Final>
__device__ __forceinline__ void stream_put_key(const StreamOut &out, const StreamPlan &pl,
                                               uint64_t key, uint64_t r, unsigned long long cnt) {
  long long kx, ky, kz;
  stream_unpack(pl, key, kx, ky, kz);
  if (Final) {
    out.keys3[3 * r] = kx;
    out.keys3[3 * r + 1] = ky;
    out.keys3[3 * r + 2] = kz;
  } else {
    out.kx[r] = kx;
    out.ky[r] = ky;
    out.kz[r] = kz;
  }
  out.cnt[r] = cnt;
}
template <bool Final>
__device__ __forceinline__ void stream_put(const StreamOut &out, uint32_t c, uint64_t r, double sum,
                                           unsigned long long cnt) {
  if (!Final) out.sum[c][r] = sum;
  else if (c < 3) out.pos[c][r] = __double2float_rn(__ddiv_rn(sum, __ull2double_rn(cnt)));
  else out.attr[c - 3][r] = __ddiv_rn(sum, __ull2double_rn(cnt));
}

// The fields of unit u of a packed point, in order: at most four, of which slot
// 0 and 2 may be f64 (then slot 1 or 3 is empty).  visit(slot, column, value).
template <class Visit>
__device__ __forceinline__ void stream_fields(const StreamLayout &lay, uint32_t u, uint4 q,
                                              Visit visit) {
#pragma unroll
  for (uint32_t h = 0; h < 2; ++h) {
    const uint32_t p = 2 * u + h;
    const uint32_t lo = h ? q.z : q.x, hi = h ? q.w : q.y;
    if (p < lay.nd) {
      visit(2 * h, lay.col_d[p], __hiloint2double(int(hi), int(lo)));
    } else {
      const uint32_t f = 2 * (p - lay.nd);
      if (f < lay.nf) visit(2 * h, lay.col_f[f], double(__uint_as_float(lo)));
      if (f + 1 < lay.nf) visit(2 * h + 1, lay.col_f[f + 1], double(__uint_as_float(hi)));
    }
  }
}

// The first value of a compensated sum: a lone one is the sum as it is; with `more` to
// follow it is Kahan::add to an empty sum, so that an infinity leaves its correction NaN
// and the sum of what follows NaN, as CompensatedSum's is.  A stream of 8M points takes
// 0.6% longer so than with a zero correction, 1.7% with add itself behind a branch.
__device__ __forceinline__ void stream_first(Kahan &k, double v, bool more) {
  const double t = __dadd_rn(0.0, v);
  k.s = more ? t : v;
  k.c = __dsub_rn(t, v);
}

// Reduces the voxel at sorted positions [i, j), one thread in sorted order, into
// output record r; v is the item at i.  A warp's voxels hold one item or a few:
// all lanes take their first item together, then loop over the rest, a group of
// columns at a time.
template <bool Records, bool Final>
__device__ __forceinline__ void stream_reduce(const SortedView &sv, const StreamPlan &pl,
                                              const StreamIn &in, const StreamOut &out,
                                              uint64_t key, uint32_t i, uint32_t j, uint32_t v,
                                              uint64_t r) {
  const bool more = j > i + 1;
  unsigned long long cnt = j - i;
  if (Records) {
    cnt = in.cnt[v];
    for (uint32_t p = i + 1; p < j; ++p) cnt += in.cnt[sv.val(p)];
  }
  stream_put_key<Final>(out, pl, key, r, cnt);
  if (Records) {
    for (uint32_t c0 = 0; c0 < in.lay.nc; c0 += 4) {
      double x[4];
      Kahan k[4];
#pragma unroll
      for (uint32_t m = 0; m < 4; ++m)
        if (c0 + m < in.lay.nc) x[m] = in.sum[c0 + m][v];
#pragma unroll
      for (uint32_t m = 0; m < 4; ++m)
        if (c0 + m < in.lay.nc) stream_first(k[m], x[m], more);
      for (uint32_t p = i + 1; p < j; ++p) {
        const uint32_t w = sv.val(p);
#pragma unroll
        for (uint32_t m = 0; m < 4; ++m)
          if (c0 + m < in.lay.nc) k[m].add(in.sum[c0 + m][w]);
      }
#pragma unroll
      for (uint32_t m = 0; m < 4; ++m)
        if (c0 + m < in.lay.nc) stream_put<Final>(out, c0 + m, r, k[m].s, cnt);
    }
    return;
  }
  const uint32_t units = in.lay.units;
  for (uint32_t u = 0; u < units; ++u) {
    Kahan k[4];
    stream_fields(in.lay, u, in.points[uint64_t(v) * units + u],
                  [&](uint32_t s, uint32_t, double x) { stream_first(k[s], x, more); });
    for (uint32_t p = i + 1; p < j; ++p)
      stream_fields(in.lay, u, in.points[uint64_t(sv.val(p)) * units + u],
                    [&](uint32_t s, uint32_t, double x) { k[s].add(x); });
    stream_fields(in.lay, u, make_uint4(0, 0, 0, 0), [&](uint32_t s, uint32_t c, double) {
      stream_put<Final>(out, c, r, k[s].s, cnt);
    });
  }
}

// Records of the voxels that start in each tile: a voxel of at most SV_SHORT
// positions is reduced by the thread holding its start; a longer one is
// queued for k_stream_long.  Thread t owns positions t, t + 256, ... of the
// tile, so that a warp's voxels, and what it writes, are consecutive.
template <bool Records, bool Final>
__global__ void __launch_bounds__(SV_THREADS, 4) k_stream_emit(Control *ctl,
                                                            SortBuffers sort,
                                                            const SortState *ss,
                                                            const StreamPlan *plan,
                                                            const uint32_t *tile_off,
                                                            const __grid_constant__ StreamIn in,
                                                            const __grid_constant__ StreamOut out,
                                                            StreamState *st,
                                                            ulonglong2 *long_list,
                                                            uint32_t long_cap) {
  constexpr int WARPS = SV_THREADS / 32;
  static_assert(SV_ITEMS * WARPS == 32, "one lane per warp row of the tile");
  __shared__ uint32_t row[SV_ITEMS * WARPS];  // voxel starts, then their prefix
  if (ld_relaxed_u32(&ctl->status)) return;
  const uint32_t n = uint32_t(ctl->n_points);
  const uint32_t tiles = (n + SV_TILE - 1) / SV_TILE;
  const SortedView sv = sorted_view(sort, *ss);
  const StreamPlan pl = *plan;
  const uint64_t flag = 1ull << pl.total_bits;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    uint64_t keys[SV_ITEMS];
    uint32_t vals[SV_ITEMS], starts[SV_ITEMS];
#pragma unroll
    for (int k = 0; k < SV_ITEMS; ++k) {
      const uint32_t i = tile * SV_TILE + k * SV_THREADS + threadIdx.x;
      bool head = false;
      keys[k] = 0;
      vals[k] = 0;
      if (i < n) {
        sv.get(i, keys[k], vals[k]);
        head = !(keys[k] & flag) && (i == 0 || sv.key(i - 1) != keys[k]);
      }
      starts[k] = __ballot_sync(FULL_MASK, head);
      if (lane == 0) row[k * WARPS + warp] = __popc(starts[k]);
    }
    __syncthreads();
    if (warp == 0) {
      uint32_t total;
      const uint32_t ex = warp_exclusive_sum(row[lane], &total);
      __syncwarp();
      row[lane] = ex;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < SV_ITEMS; ++k) {
      if (!((starts[k] >> lane) & 1u)) continue;
      const uint32_t i = tile * SV_TILE + k * SV_THREADS + threadIdx.x;
      const uint64_t slot = uint64_t(tile_off[tile]) + row[k * WARPS + warp] +
                            __popc(starts[k] & lanemask_lt());
      uint32_t j = i + 1;
      while (j < n && j - i < SV_SHORT && sv.key(j) == keys[k]) ++j;
      if (j < n && j - i == SV_SHORT && sv.key(j) == keys[k]) {
        const unsigned long long q = atomicAdd(&st->long_count, 1ull);
        if (q < long_cap) long_list[q] = make_ulonglong2(i, slot);
        else atomicOr(&ctl->status, ST_INTERNAL);
        continue;
      }
      const uint64_t r = out.base + slot;
      if (r < out.cap) stream_reduce<Records, Final>(sv, pl, in, out, keys[k], i, j, vals[k], r);
      else atomicOr(&ctl->status, ST_INTERNAL);
    }
    __syncthreads();
  }
}

// One block per queued long voxel: finds its end, then reduces every column
// with per-thread compensated sums combined in thread order.
template <bool Records, bool Final>
__global__ void __launch_bounds__(SV_THREADS) k_stream_long(Control *ctl, SortBuffers sort,
                                                            const SortState *ss,
                                                            const StreamPlan *plan,
                                                            const __grid_constant__ StreamIn in,
                                                            const __grid_constant__ StreamOut out,
                                                            const StreamState *st,
                                                            const ulonglong2 *long_list) {
  __shared__ unsigned long long end_s;
  __shared__ double red[SV_THREADS];
  __shared__ unsigned long long redc[SV_THREADS];
  if (ld_relaxed_u32(&ctl->status)) return;
  const uint32_t n = uint32_t(ctl->n_points);
  const SortedView sv = sorted_view(sort, *ss);
  const StreamPlan pl = *plan;
  const unsigned long long count = st->long_count;
  const uint32_t t = threadIdx.x;
  for (unsigned long long e = blockIdx.x; e < count; e += gridDim.x) {
    const ulonglong2 item = long_list[e];
    const uint32_t start = uint32_t(item.x);
    const uint64_t key = sv.key(start);
    if (t == 0) end_s = n;
    __syncthreads();
    for (uint32_t base = start; base < n; base += SV_THREADS) {
      const uint32_t p = base + t;
      if (p < n && sv.key(p) != key) atomicMin(&end_s, (unsigned long long)p);
      __syncthreads();
      const unsigned long long e_s = end_s;
      __syncthreads();
      if (e_s < base + SV_THREADS) break;
    }
    const uint32_t end = uint32_t(end_s);
    const uint64_t r = out.base + item.y;
    const bool ok = r < out.cap;
    unsigned long long cnt = 0;
    for (uint32_t p = start + t; p < end; p += SV_THREADS) cnt += Records ? in.cnt[sv.val(p)] : 1ull;
    redc[t] = cnt;
    __syncthreads();
    for (uint32_t w = SV_THREADS / 2; w > 0; w >>= 1) {
      if (t < w) redc[t] += redc[t + w];
      __syncthreads();
    }
    cnt = redc[0];
    if (t == 0) {
      if (ok) stream_put_key<Final>(out, pl, key, r, cnt);
      else atomicOr(&ctl->status, ST_INTERNAL);
    }
    // column c's compensated sum over the block: `mine` per thread, then in thread order
    auto column = [&](uint32_t c, const Kahan &mine) {
      red[t] = mine.s;
      __syncthreads();
      if (t == 0) {
        Kahan tot;
        for (uint32_t w = 0; w < SV_THREADS; ++w) tot.add(red[w]);
        if (ok) stream_put<Final>(out, c, r, tot.s, cnt);
      }
      __syncthreads();
    };
    if (Records) {
      for (uint32_t c = 0; c < in.lay.nc; ++c) {
        Kahan k;
        for (uint32_t p = start + t; p < end; p += SV_THREADS) k.add(in.sum[c][sv.val(p)]);
        column(c, k);
      }
    } else {
      for (uint32_t u = 0; u < in.lay.units; ++u) {
        Kahan k[4];
        uint32_t p = start + t;
        for (; p + (SV_AHEAD - 1) * SV_THREADS < end;
             p += SV_AHEAD * SV_THREADS) {
          uint4 q[SV_AHEAD];
#pragma unroll
          for (uint32_t a = 0; a < SV_AHEAD; ++a)
            q[a] = in.points[uint64_t(sv.val(p + a * SV_THREADS)) * in.lay.units + u];
#pragma unroll
          for (uint32_t a = 0; a < SV_AHEAD; ++a)
            stream_fields(in.lay, u, q[a], [&](uint32_t s, uint32_t, double x) { k[s].add(x); });
        }
        for (; p < end; p += SV_THREADS)
          stream_fields(in.lay, u, in.points[uint64_t(sv.val(p)) * in.lay.units + u],
                        [&](uint32_t s, uint32_t, double x) { k[s].add(x); });
        stream_fields(in.lay, u, make_uint4(0, 0, 0, 0),
                      [&](uint32_t s, uint32_t c, double) { column(c, k[s]); });
      }
    }
  }
}

}  // namespace srcu
