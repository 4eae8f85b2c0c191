// ransac.cuh -- RANSAC plane hypothesis scoring on the device.
//
// The reference's CPU segmenter (crates/spatialrust-segmentation/src/
// plane.rs:266-301, plane_ransac.rs:54-94) builds each hypothesis plane from
// three points in f32 (plane_from_points: cross product, normalize, d =
// -n.p0) and counts the points with |n.p + d| <= threshold (distance_xyz,
// plane.rs:39-41).  The same f32 expressions are evaluated here in the same
// order with round-to-nearest and no contraction, so every count equals the
// reference's, and so do the best hypothesis and its inlier set.
//
// Scoring is compute-bound work of n x H predicate evaluations: each thread
// keeps its points in registers, the block walks every plane held in shared
// memory, and counts go warp-reduced into shared then global counters.
#pragma once

#include "common.cuh"

namespace srcu {

constexpr int RS_THREADS = 256;
constexpr int RS_PLANES = 512;  // planes per shared-memory chunk

// What the selection leaves for the kernels after it and for the host.
struct RansacBest {
  int32_t index;      // first hypothesis of the largest count, -1: none has an inlier
  uint32_t count;
  float4 plane;
  double cnt;         // inliers counted again with the sums
  double mean[3];
};

// plane_from_points (plane_ransac.rs:79-89) in f32: invalid when |n|^2 < 1e-12.
__global__ void k_ransac_planes(const float *x, const float *y, const float *z, uint64_t n,
                                const uint32_t *hyp, uint32_t count, float4 *planes,
                                uint32_t *valid, uint32_t *counts, uint32_t *status) {
  const uint32_t h = blockIdx.x * blockDim.x + threadIdx.x;
  if (h >= count) return;
  counts[h] = 0;
  const uint32_t i0 = hyp[3 * h], i1 = hyp[3 * h + 1], i2 = hyp[3 * h + 2];
  if (i0 >= n || i1 >= n || i2 >= n) {  // cannot happen: indices are drawn below n
    atomicOr(status, ST_INTERNAL);
    planes[h] = make_float4(0.f, 0.f, 0.f, 0.f);
    valid[h] = 0;
    return;
  }
  const float p0x = x[i0], p0y = y[i0], p0z = z[i0];
  const float v1x = __fsub_rn(x[i1], p0x), v1y = __fsub_rn(y[i1], p0y), v1z = __fsub_rn(z[i1], p0z);
  const float v2x = __fsub_rn(x[i2], p0x), v2y = __fsub_rn(y[i2], p0y), v2z = __fsub_rn(z[i2], p0z);
  // Vec3::cross (crates/spatialrust-math/src/vec.rs:71-78)
  float nx = __fsub_rn(__fmul_rn(v1y, v2z), __fmul_rn(v1z, v2y));
  float ny = __fsub_rn(__fmul_rn(v1z, v2x), __fmul_rn(v1x, v2z));
  float nz = __fsub_rn(__fmul_rn(v1x, v2y), __fmul_rn(v1y, v2x));
  const float ls = __fadd_rn(__fadd_rn(__fmul_rn(nx, nx), __fmul_rn(ny, ny)), __fmul_rn(nz, nz));
  if (ls < 1e-12f) {  // no plane (a NaN length goes on and counts no inlier)
    planes[h] = make_float4(0.f, 0.f, 0.f, 0.f);
    valid[h] = 0;
    return;
  }
  // Vec3::normalize (vec.rs:94-100): x / sqrt(x.x)
  const float len = __fsqrt_rn(ls);
  nx = __fdiv_rn(nx, len);
  ny = __fdiv_rn(ny, len);
  nz = __fdiv_rn(nz, len);
  const float dot = __fadd_rn(__fadd_rn(__fmul_rn(nx, p0x), __fmul_rn(ny, p0y)), __fmul_rn(nz, p0z));
  planes[h] = make_float4(nx, ny, nz, -dot);
  valid[h] = 1;
}

// PlaneModel::distance_xyz (plane.rs:39-41) <= threshold, in the reference's order.
__device__ __forceinline__ bool plane_inlier(float4 pl, float px, float py, float pz, float thr) {
  const float s = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(pl.x, px), __fmul_rn(pl.y, py)),
                                      __fmul_rn(pl.z, pz)),
                            pl.w);
  return fabsf(s) <= thr;
}

// Packed f32x2 arithmetic: two IEEE round-to-nearest operations, one per half.  A product
// is written as a fused multiply-add of -0, which rounds it and keeps its sign: the
// assembler fuses mul.rn.f32x2 with an add.rn.f32x2 that follows, explicit rounding or
// not, and the sum is then not the reference's (over georeferenced coordinates counts
// went wrong by hundreds).  The zero comes as a kernel argument, out of its sight.
__device__ __forceinline__ uint64_t rs_pack(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ uint64_t rs_mul(uint64_t a, uint64_t b, uint64_t minus_zero) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(minus_zero));
  return r;
}
__device__ __forceinline__ uint64_t rs_add(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
constexpr uint64_t RS_MINUS_ZERO = 0x8000000080000000ull;  // (-0, -0)

// counts[h] += inliers of plane h among this block's points, for the planes
// [blockIdx.y * per_chunk, +per_chunk): the second grid dimension splits the
// hypotheses so that small clouds fill every SM.
//
// plane_inlier's operations in its order, on two points at a time: six packed
// instructions for what takes twelve apart, which leaves the comparison and the
// count.  PAIRS pairs of points per thread share each plane's loads, its warp
// reduction and its shared-memory atomic.  460k points x 1000 planes: 142 us,
// 179 us with scalar arithmetic and eight points per thread.
template <int PAIRS>
__global__ void __launch_bounds__(RS_THREADS) k_ransac_score(const float *x, const float *y,
                                                             const float *z, uint64_t n,
                                                             const float4 *planes, uint32_t count,
                                                             uint32_t per_chunk, float thr,
                                                             uint64_t minus_zero,
                                                             uint32_t *counts) {
  __shared__ ulonglong2 sp[RS_PLANES][2];  // (a, a) (b, b) / (c, c) (d, d)
  __shared__ uint32_t sc[RS_PLANES];
  uint64_t px[PAIRS], py[PAIRS], pz[PAIRS];
  const uint64_t first = uint64_t(blockIdx.x) * (RS_THREADS * 2 * PAIRS);
#pragma unroll
  for (int k = 0; k < PAIRS; ++k) {
    const uint64_t i = first + uint64_t(2 * k) * RS_THREADS + threadIdx.x;  // coalesced
    const uint64_t j = i + RS_THREADS;
    const float nanv = __int_as_float(0x7fc00000);  // NaN: never an inlier
    px[k] = rs_pack(i < n ? x[i] : nanv, j < n ? x[j] : nanv);
    py[k] = rs_pack(i < n ? y[i] : 0.f, j < n ? y[j] : 0.f);
    pz[k] = rs_pack(i < n ? z[i] : 0.f, j < n ? z[j] : 0.f);
  }
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t c_begin = blockIdx.y * per_chunk;
  const uint32_t c_end = min(count, c_begin + per_chunk);
  for (uint32_t c0 = c_begin; c0 < c_end; c0 += RS_PLANES) {
    const uint32_t m = min(uint32_t(RS_PLANES), c_end - c0);
    for (uint32_t j = threadIdx.x; j < m; j += RS_THREADS) {
      const float4 pl = planes[c0 + j];
      sp[j][0] = make_ulonglong2(rs_pack(pl.x, pl.x), rs_pack(pl.y, pl.y));
      sp[j][1] = make_ulonglong2(rs_pack(pl.z, pl.z), rs_pack(pl.w, pl.w));
      sc[j] = 0;
    }
    __syncthreads();
#pragma unroll 2
    for (uint32_t j = 0; j < m; ++j) {
      const ulonglong2 ab = sp[j][0], cd = sp[j][1];
      uint32_t c = 0;
#pragma unroll
      for (int k = 0; k < PAIRS; ++k) {
        const uint64_t s =
            rs_add(rs_add(rs_add(rs_mul(ab.x, px[k], minus_zero), rs_mul(ab.y, py[k], minus_zero)),
                          rs_mul(cd.x, pz[k], minus_zero)),
                   cd.y);
        float s0, s1;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(s0), "=f"(s1) : "l"(s));
        c += fabsf(s0) <= thr ? 1u : 0u;
        c += fabsf(s1) <= thr ? 1u : 0u;
      }
      c = __reduce_add_sync(FULL_MASK, c);
      if (lane == 0 && c) atomicAdd(&sc[j], c);
    }
    __syncthreads();
    for (uint32_t j = threadIdx.x; j < m; j += RS_THREADS)
      if (sc[j]) atomicAdd(&counts[c0 + j], sc[j]);
    __syncthreads();
  }
}

// The CPU loop's choice: a candidate replaces the best only with strictly more
// inliers, so the first hypothesis of the largest count.  One block of 1024.
__global__ void __launch_bounds__(1024) k_ransac_best(const float4 *planes, const uint32_t *valid,
                                                      const uint32_t *counts, uint32_t count,
                                                      RansacBest *best) {
  __shared__ unsigned long long red[32];
  unsigned long long key = 0;  // (count, ~index): larger counts, then earlier hypotheses
  for (uint32_t h = threadIdx.x; h < count; h += 1024)
    if (valid[h] && counts[h]) {
      const unsigned long long k = ((unsigned long long)counts[h] << 32) | (0xffffffffu - h);
      key = k > key ? k : key;
    }
  for (int round = 0; round < 2; ++round) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long k = __shfl_xor_sync(FULL_MASK, key, o);
      key = k > key ? k : key;
    }
    if (round) break;
    if ((threadIdx.x & 31u) == 0) red[threadIdx.x >> 5] = key;
    __syncthreads();
    key = red[threadIdx.x & 31u];
  }
  if (threadIdx.x == 0) {
    const uint32_t h = 0xffffffffu - uint32_t(key);
    best->index = key ? int32_t(h) : -1;
    best->count = uint32_t(key >> 32);
    best->plane = key ? planes[h] : make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

// Inlier mask of the best plane, and per-block FP64 partial sums over the
// inliers: pass 0: count, sum x, y, z; pass 1 (with the mean): the six centred
// second moments (refine_plane_from_inliers, plane_ransac.rs:96-150).  Blocks sum
// in a fixed order, so the result does not depend on scheduling.  Does nothing
// where the segmentation fails for want of inliers.
constexpr int RM_THREADS = 256;

__global__ void __launch_bounds__(RM_THREADS) k_ransac_moments(const float *x, const float *y,
                                                               const float *z, uint64_t n,
                                                               const RansacBest *best,
                                                               unsigned long long min_inliers,
                                                               float thr, uint8_t *mask, int pass,
                                                               double *partials) {
  __shared__ double red[6][RM_THREADS];
  if (best->index < 0 || best->count < min_inliers) return;
  const float4 pl = best->plane;
  const double mx = best->mean[0], my = best->mean[1], mz = best->mean[2];  // pass 1
  double acc[6] = {0, 0, 0, 0, 0, 0};
  for (uint64_t i = blockIdx.x * uint64_t(RM_THREADS) + threadIdx.x; i < n;
       i += uint64_t(gridDim.x) * RM_THREADS) {
    const float px = x[i], py = y[i], pz = z[i];
    const bool in = plane_inlier(pl, px, py, pz, thr);
    if (pass == 0) {
      if (mask) mask[i] = in ? 1 : 0;
      if (in) {
        acc[0] += 1.0;
        acc[1] += double(px);
        acc[2] += double(py);
        acc[3] += double(pz);
      }
    } else if (in) {
      const double dx = double(px) - mx, dy = double(py) - my, dz = double(pz) - mz;
      acc[0] += dx * dx;
      acc[1] += dy * dy;
      acc[2] += dz * dz;
      acc[3] += dx * dy;
      acc[4] += dx * dz;
      acc[5] += dy * dz;
    }
  }
  const int t = threadIdx.x;
#pragma unroll
  for (int k = 0; k < 6; ++k) red[k][t] = acc[k];
  __syncthreads();
  for (int w = RM_THREADS / 2; w >= 32; w >>= 1) {
    if (t < w) {
#pragma unroll
      for (int k = 0; k < 6; ++k) red[k][t] += red[k][t + w];
    }
    __syncthreads();
  }
  if (t < 32) {
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      double v = red[k][t];
#pragma unroll
      for (int w = 16; w > 0; w >>= 1) v += __shfl_down_sync(FULL_MASK, v, w);
      if (t == 0) partials[blockIdx.x * 6 + k] = v;
    }
  }
}

// Count and mean from pass 0's partial sums, in block order.  One block of 32 * k
// threads; at most RM_MAX_BLOCKS partials.
constexpr uint32_t RM_MAX_BLOCKS = 512;
__global__ void __launch_bounds__(256) k_ransac_mean(const double *partials, uint32_t blocks,
                                                     unsigned long long min_inliers,
                                                     RansacBest *best) {
  __shared__ double s[4][RM_MAX_BLOCKS];
  __shared__ double sum[4];
  if (best->index < 0 || best->count < min_inliers) return;
  for (uint32_t b = threadIdx.x; b < blocks; b += 256)
    for (int k = 0; k < 4; ++k) s[k][b] = partials[b * 6 + k];
  __syncthreads();
  if (threadIdx.x < 4) {
    double v = 0;
#pragma unroll 8
    for (uint32_t b = 0; b < blocks; ++b) v += s[threadIdx.x][b];
    sum[threadIdx.x] = v;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    best->cnt = sum[0];
    for (int a = 0; a < 3; ++a) best->mean[a] = __ddiv_rn(sum[1 + a], sum[0]);
  }
}

}  // namespace srcu
