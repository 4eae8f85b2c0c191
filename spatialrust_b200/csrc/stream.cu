// stream.cu -- host side of the bounded streaming voxel (srcu_stream_voxel_*,
// include/srcuda.h).  Included at the end of srcuda.cu: it drives the
// context's sort buffers and control block like the other chains.
//
// Mirrors StreamingVoxelSource::try_build / next_chunk
// (crates/spatialrust-pipeline/src/streaming.rs:414-535, 594-676):
//   push()    packs a chunk into the device run buffer; a full buffer is a run:
//             bounds -> plan -> onesweep sort -> segment reduction into partial
//             records (key, count, compensated FP64 column sums);
//   finish()  reduces the last run, checks the reference's run and spool
//             limits, sorts every partial record by key and reduces again; the
//             only run of a short stream is reduced into the outputs directly;
//   fetch()   copies a window of the final voxels (next_chunk's chunks).
#include "stream.cuh"

struct srcu_stream_voxel {
  srcu_ctx *ctx = nullptr;
  srcu_stream_voxel_params prm{};
  uint32_t nc = 3;
  double leaf = 0.0;
  uint64_t dev_run = 0;   // points per device run
  uint64_t fill = 0;      // points of the run so far, the last `staged` of them unpacked
  uint64_t staged = 0;    // points in the staging columns
  uint64_t stage_cap = 0; // points they hold
  uint64_t points = 0;    // points pushed
  uint64_t device_runs = 0;
  uint64_t records = 0;   // partial records stored
  uint64_t rec_cap = 0;
  uint64_t voxels = 0;
  bool finished = false;
  StreamLayout lay{};
  int occ_point[2] = {1, 1}, occ_record[2] = {1, 1};  // by kStreamSort shape
  DevBuf run;                                  // run buffer: packed points
  DevBuf stage[MAX_COLS];                      // columns of a chunk not read in place
  DevBuf rk[3], rcnt, rsum[MAX_COLS];          // partial records
  DevBuf opos[3], oattr[MAX_COLS], okeys, ocnt; // finished outputs
  DevBuf tile_heads, tile_off, long_list, plan, state;
  StreamState *state_host = nullptr;           // pinned
};

namespace {

// Points of a chunk staged at a time, and points that small chunks gather to before they
// are packed.  A kernel for every push makes it longer (1000 host points with nine f64
// attributes 50 us, 46 gathered; 16384 with two 60, 50 gathered).
constexpr uint64_t kStreamStage = uint64_t(1) << 20;
constexpr uint64_t kStreamGather = uint64_t(1) << 16;

uint32_t sv_elem(const srcu_stream_voxel *sv, uint32_t c) {
  return (c >= 3 && ((sv->prm.attr_f64_mask >> (c - 3)) & 1u)) ? 8u : 4u;
}

// Grows a device buffer to `bytes`, keeping its first `keep` bytes.
srcu_status grow_keep(srcu_ctx *ctx, DevBuf &b, size_t bytes, size_t keep) {
  if (b.bytes >= bytes) return SRCU_OK;
  DevBuf nb;
  ST_TRY(ensure(ctx, nb, bytes));
  if (keep && b.p) CU_TRY(cudaMemcpyAsync(nb.p, b.p, keep, cudaMemcpyDeviceToDevice, ctx->stream));
  if (b.p) {
    CU_TRY(cudaStreamSynchronize(ctx->stream));
    release(ctx, b);
  }
  b = nb;
  return SRCU_OK;
}

srcu_status sv_reserve_records(srcu_stream_voxel *sv, uint64_t need) {
  if (need <= sv->rec_cap) return SRCU_OK;
  srcu_ctx *ctx = sv->ctx;
  const uint64_t cap = std::max<uint64_t>({need, 2 * sv->rec_cap, 4 * sv->dev_run});
  const size_t keep = size_t(sv->records) * 8;
  for (int a = 0; a < 3; ++a) ST_TRY(grow_keep(ctx, sv->rk[a], cap * 8, keep));
  ST_TRY(grow_keep(ctx, sv->rcnt, cap * 8, keep));
  for (uint32_t c = 0; c < sv->nc; ++c) ST_TRY(grow_keep(ctx, sv->rsum[c], cap * 8, keep));
  sv->rec_cap = cap;
  return SRCU_OK;
}

// The f64 columns first, then the f32 ones in pairs, in 16-byte units.
void sv_layout(srcu_stream_voxel *sv) {
  StreamLayout &l = sv->lay;
  l = StreamLayout{};
  l.nc = sv->nc;
  for (uint32_t c = 0; c < sv->nc; ++c)
    if (sv_elem(sv, c) == 8) l.col_d[l.nd++] = c;
    else l.col_f[l.nf++] = c;
  l.units = (l.nd + (l.nf + 1) / 2 + 1) / 2;
}

StreamOut sv_partial_out(srcu_stream_voxel *sv) {
  StreamOut o{};
  o.kx = ptr<long long>(sv->rk[0]);
  o.ky = ptr<long long>(sv->rk[1]);
  o.kz = ptr<long long>(sv->rk[2]);
  o.cnt = ptr<unsigned long long>(sv->rcnt);
  for (uint32_t c = 0; c < sv->nc; ++c) o.sum[c] = ptr<double>(sv->rsum[c]);
  o.base = sv->records;
  o.cap = sv->rec_cap;
  return o;
}

// The outputs, for up to r voxels.
srcu_status sv_final_out(srcu_stream_voxel *sv, uint64_t r, StreamOut &o) {
  srcu_ctx *ctx = sv->ctx;
  for (int a = 0; a < 3; ++a) ST_TRY(ensure(ctx, sv->opos[a], r * 4));
  for (uint32_t c = 3; c < sv->nc; ++c) ST_TRY(ensure(ctx, sv->oattr[c], r * 8));
  ST_TRY(ensure(ctx, sv->okeys, r * 24));
  ST_TRY(ensure(ctx, sv->ocnt, r * 8));
  o = StreamOut{};
  for (int a = 0; a < 3; ++a) o.pos[a] = ptr<float>(sv->opos[a]);
  for (uint32_t c = 3; c < sv->nc; ++c) o.attr[c - 3] = ptr<double>(sv->oattr[c]);
  o.keys3 = ptr<long long>(sv->okeys);
  o.cnt = ptr<unsigned long long>(sv->ocnt);
  o.cap = r;
  return SRCU_OK;
}

// The streams' sorts run in two of the sort's launch shapes whatever tuning a context
// has: 8 keys per thread x 3 blocks of 256 threads up to 441k keys, 8 x 2 x 512 with
// 9-bit digits above (16 x 2 x 256, used for all before: 4.2M points 238 us, 205 us
// here).  The voxel sort's built-in table has another shape between 623k and 882k keys.
constexpr int kStreamSort[2] = {1, 6};
constexpr uint64_t kStreamSortSmall = 441000;

template <class Src>
srcu_status sv_sort(srcu_stream_voxel *sv, const Src &src, uint64_t n, const int (&occ)[2]) {
  srcu_ctx *ctx = sv->ctx;
  Launch l(ctx, SRCU_K_VOXEL_SORT);
  const SortBuffers sb = sort_buffers(ctx);
  const bool large = n > kStreamSortSmall;
  const uint32_t cap = uint32_t(ctx->num_sms) * uint32_t(occ[large]);
  CU_TRY((large ? launch_sort_config<Src, kStreamSort[1]>
                : launch_sort_config<Src, kStreamSort[0]>)(ctx->stream, cap, src, ctx->ctl,
                                                           ctx->ctl->hist_v, sb, EP_VSORT, WK_VSORT,
                                                           &ctx->ctl->vsort, n));
  return SRCU_OK;
}

// Segment reduction of the current sort (ctl->n_points = n sorted items).
template <bool Records, bool Final>
srcu_status sv_reduce(srcu_stream_voxel *sv, uint64_t n, const StreamIn &in, const StreamOut &out,
                      int count_finite) {
  srcu_ctx *ctx = sv->ctx;
  const uint64_t tiles = std::max<uint64_t>(1, ceil_div(n, SV_TILE));
  const uint64_t long_cap = n / (SV_SHORT + 1) + 1;
  ST_TRY(ensure(ctx, sv->tile_heads, tiles * 4));
  ST_TRY(ensure(ctx, sv->tile_off, tiles * 4));
  ST_TRY(ensure(ctx, sv->long_list, long_cap * sizeof(ulonglong2)));
  const uint32_t grid = std::max<uint32_t>(
      1, std::min<uint32_t>(uint32_t(tiles), uint32_t(ctx->num_sms) * 8));
  StreamState *st = ptr<StreamState>(sv->state);
  const StreamPlan *pl = ptr<const StreamPlan>(sv->plan);
  Launch l(ctx, SRCU_K_VOXEL_SEGMENTS, 4);
  k_stream_flags<<<grid, SV_THREADS, 0, ctx->stream>>>(ctx->ctl, sort_buffers(ctx), &ctx->ctl->vsort,
                                                       pl, ptr<uint32_t>(sv->tile_heads), st,
                                                       count_finite);
  k_stream_scan<<<1, 1024, 0, ctx->stream>>>(ctx->ctl, ptr<const uint32_t>(sv->tile_heads),
                                             ptr<uint32_t>(sv->tile_off), st);
  k_stream_emit<Records, Final><<<grid, SV_THREADS, 0, ctx->stream>>>(
      ctx->ctl, sort_buffers(ctx), &ctx->ctl->vsort, pl, ptr<const uint32_t>(sv->tile_off), in, out,
      st, ptr<ulonglong2>(sv->long_list), uint32_t(std::min<uint64_t>(long_cap, 0xffffffffu)));
  k_stream_long<Records, Final><<<uint32_t(ctx->num_sms) * 2, SV_THREADS, 0, ctx->stream>>>(
      ctx->ctl, sort_buffers(ctx), &ctx->ctl->vsort, pl, in, out, st,
      ptr<const ulonglong2>(sv->long_list));
  CU_TRY(cudaGetLastError());
  return SRCU_OK;
}

// Reads the stream state and the control block; maps a key overflow to the
// reference's error text when the key left the i64 range.
srcu_status sv_sync(srcu_stream_voxel *sv) {
  srcu_ctx *ctx = sv->ctx;
  CU_TRY(cudaMemcpyAsync(sv->state_host, sv->state.p, sizeof(StreamState), cudaMemcpyDeviceToHost,
                         ctx->stream));
  srcu_status s = read_control(ctx);
  if (s == SRCU_ERR_KEY_OVERFLOW) {
    if (sv->state_host->overflow == 1)
      return fail(ctx, SRCU_ERR_INVALID_ARGUMENT, "voxel coordinate exceeds signed 64-bit range");
    return fail(ctx, SRCU_ERR_KEY_OVERFLOW,
                "the stream's voxel keys span more than 63 bits when packed");
  }
  return s;
}

// Columns of n points -> records of the run from point `at` on.
srcu_status sv_pack(srcu_stream_voxel *sv, const StreamChunk &ch, uint64_t at, uint64_t n) {
  srcu_ctx *ctx = sv->ctx;
  const uint32_t grid = std::min<uint32_t>(ceil_div(n, 256), uint32_t(ctx->num_sms) * 8);
  k_stream_pack<<<grid, 256, 0, ctx->stream>>>(ch, sv->lay, n,
                                               ptr<uint4>(sv->run) + at * sv->lay.units);
  CU_TRY(cudaGetLastError());
  return SRCU_OK;
}

srcu_status sv_pack_staged(srcu_stream_voxel *sv) {
  const uint64_t n = sv->staged;
  if (n == 0) return SRCU_OK;
  StreamChunk ch{};
  for (uint32_t c = 0; c < sv->nc; ++c) ch.col[c] = sv->stage[c].p;
  sv->staged = 0;
  return sv_pack(sv, ch, sv->fill - n, n);
}

// Copies n points of a chunk (its columns from point `first` on) behind the staged ones.
srcu_status sv_stage(srcu_stream_voxel *sv, const void *const *src, uint64_t first, uint64_t n,
                     cudaMemcpyKind kind) {
  srcu_ctx *ctx = sv->ctx;
  if (sv->staged + n > sv->stage_cap) {
    ST_TRY(sv_pack_staged(sv));
    if (n > sv->stage_cap) {
      const uint64_t cap = std::max(n, std::min(kStreamGather, sv->dev_run));
      sv->stage_cap = 0;
      for (uint32_t c = 0; c < sv->nc; ++c) ST_TRY(ensure(ctx, sv->stage[c], cap * sv_elem(sv, c)));
      sv->stage_cap = cap;
    }
  }
  for (uint32_t c = 0; c < sv->nc; ++c) {
    const uint32_t e = sv_elem(sv, c);
    CU_TRY(cudaMemcpyAsync(ptr<char>(sv->stage[c]) + sv->staged * e,
                           static_cast<const char *>(src[c]) + first * e, n * e, kind, ctx->stream));
  }
  sv->staged += n;
  return SRCU_OK;
}

// Sorts and reduces the run buffer into partial records, or, as the stream's only
// run, into the outputs.
template <bool Final>
srcu_status sv_flush(srcu_stream_voxel *sv) {
  const uint64_t n = sv->fill;
  if (n == 0) return SRCU_OK;
  ST_TRY(sv_pack_staged(sv));
  srcu_ctx *ctx = sv->ctx;
  StreamOut out{};
  if (Final) {
    ST_TRY(sv_final_out(sv, n, out));
  } else {
    ST_TRY(sv_reserve_records(sv, sv->records + n));
    out = sv_partial_out(sv);
  }
  ST_TRY(reserve(ctx, n, 0, false, false, false));
  ST_TRY(reserve_batch(ctx, 1));
  const Batch bt = make_batch(ctx, 1);
  ST_TRY(begin_chain(ctx, n, bt, 1, nullptr, nullptr));
  const uint4 *points = ptr<const uint4>(sv->run);
  {
    Launch l(ctx, SRCU_K_BOUNDS);
    const uint32_t grid = std::max<uint32_t>(1, std::min<uint32_t>(ceil_div(n, 256),
                                                                    uint32_t(ctx->num_sms) * 8));
    k_stream_bounds<<<grid, 256, 0, ctx->stream>>>(ctx->ctl, points, sv->lay, bt.bounds);
  }
  {
    Launch l(ctx, SRCU_K_VOXEL_PLAN);
    k_stream_plan<<<1, 32, 0, ctx->stream>>>(ctx->ctl, bt.bounds, sv->leaf,
                                             ptr<StreamPlan>(sv->plan), ptr<StreamState>(sv->state));
  }
  StreamPointSrc src{};
  src.points = points;
  src.lay = sv->lay;
  src.plan_ptr = ptr<const StreamPlan>(sv->plan);
  src.leaf = sv->leaf;
  ST_TRY(sv_sort(sv, src, n, sv->occ_point));
  StreamIn in{};
  in.points = points;
  in.lay = sv->lay;
  ST_TRY((sv_reduce<false, Final>(sv, n, in, out, 1)));
  ST_TRY(sv_sync(sv));
  sv->records += sv->state_host->segments;
  sv->device_runs += 1;
  sv->fill = 0;
  return SRCU_OK;
}

srcu_status sv_finish(srcu_stream_voxel *sv) {
  srcu_ctx *ctx = sv->ctx;
  const bool one_run = sv->device_runs == 0;
  ST_TRY(one_run ? sv_flush<true>(sv) : sv_flush<false>(sv));
  // The reference spills every finite point into runs of run_points
  // (streaming.rs:458-485): its run count and spool extent follow from the
  // finite-point count alone, and so do its two fail-closed limits.  (The
  // last run's flush read the state back.)
  const uint64_t finite = sv->state_host->finite;
  const uint64_t runs = (finite + sv->prm.run_points - 1) / sv->prm.run_points;
  if (runs > sv->prm.max_runs)
    return fail(ctx, SRCU_ERR_INVALID_ARGUMENT, "streaming voxel run limit %llu exceeded",
                (unsigned long long)sv->prm.max_runs);
  const uint64_t spool = runs * 8 + finite * (32 + 8 * uint64_t(sv->nc));
  if (sv->prm.spool_limit_bytes && spool > sv->prm.spool_limit_bytes)
    return fail(ctx, SRCU_ERR_INVALID_ARGUMENT, "spool limit exceeded: requested extent %llu, limit %llu",
                (unsigned long long)spool, (unsigned long long)sv->prm.spool_limit_bytes);
  const uint64_t r = sv->records;
  sv->voxels = 0;
  if (r == 0) return SRCU_OK;
  if (r > LB_MAX_COUNT)
    return fail(ctx, SRCU_ERR_INVALID_ARGUMENT, "%llu partial voxel records exceed the merge limit %llu",
                (unsigned long long)r, (unsigned long long)LB_MAX_COUNT);
  if (one_run) {
    sv->voxels = r;
    return SRCU_OK;
  }
  StreamOut out{};
  ST_TRY(sv_final_out(sv, r, out));
  ST_TRY(reserve(ctx, r, 0, false, false, false));
  ST_TRY(reserve_batch(ctx, 1));
  ST_TRY(begin_chain(ctx, r, make_batch(ctx, 1), 1, nullptr, nullptr));
  {
    Launch l(ctx, SRCU_K_VOXEL_PLAN);
    k_stream_merge_plan<<<1, 32, 0, ctx->stream>>>(ctx->ctl, ptr<StreamPlan>(sv->plan),
                                                   ptr<StreamState>(sv->state));
  }
  StreamRecordSrc src{};
  src.kx = ptr<const long long>(sv->rk[0]);
  src.ky = ptr<const long long>(sv->rk[1]);
  src.kz = ptr<const long long>(sv->rk[2]);
  src.plan_ptr = ptr<const StreamPlan>(sv->plan);
  ST_TRY(sv_sort(sv, src, r, sv->occ_record));
  StreamIn in{};
  in.lay = sv->lay;
  in.cnt = ptr<const unsigned long long>(sv->rcnt);
  for (uint32_t c = 0; c < sv->nc; ++c) in.sum[c] = ptr<const double>(sv->rsum[c]);
  ST_TRY((sv_reduce<true, true>(sv, r, in, out, 0)));
  CU_TRY(cudaGetLastError());
  ST_TRY(sv_sync(sv));
  sv->voxels = sv->state_host->segments;
  return SRCU_OK;
}

void sv_release(srcu_stream_voxel *sv) {
  srcu_ctx *ctx = sv->ctx;
  for (auto &b : sv->stage) release(ctx, b);
  for (auto &b : sv->rk) release(ctx, b);
  for (auto &b : sv->rsum) release(ctx, b);
  for (auto &b : sv->opos) release(ctx, b);
  for (auto &b : sv->oattr) release(ctx, b);
  DevBuf *rest[] = {&sv->run, &sv->rcnt, &sv->ocnt, &sv->okeys, &sv->tile_heads, &sv->tile_off,
                    &sv->long_list, &sv->plan, &sv->state};
  for (DevBuf *b : rest) release(ctx, *b);
}

}  // namespace

extern "C" {

srcu_status srcu_stream_voxel_create(srcu_ctx *ctx, const srcu_stream_voxel_params *params,
                                     srcu_stream_voxel **out) {
  if (!ctx || !out) return SRCU_ERR_INVALID_ARGUMENT;
  *out = nullptr;
  if (!params) return fail(ctx, SRCU_ERR_INVALID_ARGUMENT, "stream params are NULL");
  // StreamingVoxelConfig::new (streaming.rs:345-363)
  if (!(params->leaf_size > 0.0f) || params->leaf_size == INFINITY)
    return fail(ctx, SRCU_ERR_INVALID_ARGUMENT, "streaming voxel leaf size must be positive and finite");
  if (params->run_points == 0 || params->max_runs == 0)
    return fail(ctx, SRCU_ERR_INVALID_ARGUMENT,
                "streaming voxel run_points and max_runs must be positive");
  if (params->n_attrs > MAX_COLS - 3)
    return fail(ctx, SRCU_ERR_INVALID_ARGUMENT, "at most %d attribute columns are supported",
                MAX_COLS - 3);
  CU_TRY(cudaSetDevice(ctx->device));
  // Reuse the buffers of the context's last stream: a new stream then
  // allocates nothing until it outgrows them.
  srcu_stream_voxel *sv = ctx->parked_stream;
  ctx->parked_stream = nullptr;
  if (!sv) sv = new srcu_stream_voxel();
  sv->ctx = ctx;
  sv->prm = *params;
  sv->nc = 3 + params->n_attrs;
  sv->leaf = double(params->leaf_size);
  sv->fill = sv->points = sv->device_runs = sv->records = sv->voxels = 0;
  // re-derived from the kept buffers' sizes as points and records arrive
  sv->staged = sv->stage_cap = sv->rec_cap = 0;
  sv->finished = false;
  // By default a device run holds at least 2^22 points whatever run_points
  // is: the run size only partitions the sums, the voxels do not depend on it,
  // and larger runs sort more efficiently and synchronise less often.
  sv->dev_run = params->device_run_points
                    ? uint64_t(params->device_run_points)
                    : std::max<uint64_t>(params->run_points, uint64_t(1) << 22);
  sv->dev_run = std::min<uint64_t>(sv->dev_run, uint64_t(1) << 26);
  auto bail = [&](srcu_status st) {
    stream_voxel_free(sv);
    return st;
  };
  sv_layout(sv);
  if (sort_config_setup<StreamPointSrc, kStreamSort[0]>(&sv->occ_point[0]) != cudaSuccess ||
      sort_config_setup<StreamPointSrc, kStreamSort[1]>(&sv->occ_point[1]) != cudaSuccess ||
      sort_config_setup<StreamRecordSrc, kStreamSort[0]>(&sv->occ_record[0]) != cudaSuccess ||
      sort_config_setup<StreamRecordSrc, kStreamSort[1]>(&sv->occ_record[1]) != cudaSuccess)
    return bail(fail(ctx, SRCU_ERR_CUDA, "cannot configure the streaming sort kernels"));
  srcu_status s = ensure(ctx, sv->run, sv->dev_run * sv->lay.units * 16);
  if (s == SRCU_OK) s = ensure(ctx, sv->plan, sizeof(StreamPlan));
  if (s == SRCU_OK) s = ensure(ctx, sv->state, sizeof(StreamState));
  if (s != SRCU_OK) return bail(s);
  if (!sv->state_host &&
      cudaMallocHost(reinterpret_cast<void **>(&sv->state_host), sizeof(StreamState)) != cudaSuccess)
    return bail(fail(ctx, SRCU_ERR_CUDA, "cannot allocate pinned stream state"));
  StreamState init{};
  for (int a = 0; a < 3; ++a) {
    init.gmin[a] = LLONG_MAX;
    init.gmax[a] = LLONG_MIN;
  }
  *sv->state_host = init;
  if (cudaMemcpyAsync(sv->state.p, sv->state_host, sizeof(StreamState), cudaMemcpyHostToDevice,
                      ctx->stream) != cudaSuccess ||
      cudaStreamSynchronize(ctx->stream) != cudaSuccess)
    return bail(fail(ctx, SRCU_ERR_CUDA, "cannot initialise the stream state"));
  *out = sv;
  return SRCU_OK;
}

srcu_status srcu_stream_voxel_push(srcu_stream_voxel *sv, const srcu_cloud *chunk) {
  if (!sv) return SRCU_ERR_INVALID_ARGUMENT;
  srcu_ctx *ctx = sv->ctx;
  ST_TRY(check_cloud(ctx, chunk));
  if (sv->finished) return fail(ctx, SRCU_ERR_INVALID_ARGUMENT, "the stream is already finished");
  if (chunk->n_attrs != sv->prm.n_attrs)
    return fail(ctx, SRCU_ERR_INVALID_ARGUMENT, "chunk has %u attribute columns, the stream %u",
                chunk->n_attrs, sv->prm.n_attrs);
  if (strided(chunk))
    return fail(ctx, SRCU_ERR_INVALID_ARGUMENT, "streaming voxel chunks must be packed columns");
  CU_TRY(cudaSetDevice(ctx->device));
  const void *src[MAX_COLS] = {chunk->x, chunk->y, chunk->z};
  for (uint32_t a = 0; a < chunk->n_attrs; ++a) src[3 + a] = chunk->attrs[a];
  // device columns are read where they are, unless one is not aligned to its elements or
  // not in memory that a kernel may read: a chunk with such a column is staged by copies
  const cudaMemcpyKind kind = chunk->on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
  bool in_place = chunk->on_device != 0;
  for (uint32_t c = 0; c < sv->nc; ++c)
    in_place = in_place && reinterpret_cast<uintptr_t>(src[c]) % sv_elem(sv, c) == 0 &&
               (chunk->n == 0 || own_memory(ctx, src[c]));
  uint64_t done = 0;
  while (done < chunk->n) {
    uint64_t take = std::min<uint64_t>(chunk->n - done, sv->dev_run - sv->fill);
    if (!in_place) take = std::min(take, kStreamStage);
    if (take && in_place) {
      ST_TRY(sv_pack_staged(sv));
      StreamChunk ch{};
      for (uint32_t c = 0; c < sv->nc; ++c)
        ch.col[c] = static_cast<const char *>(src[c]) + done * sv_elem(sv, c);
      ST_TRY(sv_pack(sv, ch, sv->fill, take));
    } else if (take) {
      ST_TRY(sv_stage(sv, src, done, take, kind));
    }
    sv->fill += take;
    done += take;
    if (sv->fill == sv->dev_run) ST_TRY(sv_flush<false>(sv));
  }
  sv->points += chunk->n;
  CU_TRY(cudaStreamSynchronize(ctx->stream));  // the chunk's memory may be reused on return
  return SRCU_OK;
}

srcu_status srcu_stream_voxel_finish(srcu_stream_voxel *sv, srcu_stream_voxel_info *info) {
  if (!sv) return SRCU_ERR_INVALID_ARGUMENT;
  srcu_ctx *ctx = sv->ctx;
  if (info) memset(info, 0, sizeof(*info));
  if (sv->finished) return fail(ctx, SRCU_ERR_INVALID_ARGUMENT, "the stream is already finished");
  CU_TRY(cudaSetDevice(ctx->device));
  sv->finished = true;
  ST_TRY(sv_finish(sv));
  if (info) {
    const uint64_t finite = sv->state_host->finite;
    info->points = sv->points;
    info->finite_points = finite;
    info->runs = (finite + sv->prm.run_points - 1) / sv->prm.run_points;
    info->spool_bytes = info->runs * 8 + finite * (32 + 8 * uint64_t(sv->nc));
    info->device_runs = sv->device_runs;
    info->partial_records = sv->records;
    info->voxels = sv->voxels;
  }
  return SRCU_OK;
}

srcu_status srcu_stream_voxel_fetch(srcu_stream_voxel *sv, uint64_t first, uint64_t count,
                                    const srcu_stream_voxel_out *out) {
  if (!sv) return SRCU_ERR_INVALID_ARGUMENT;
  srcu_ctx *ctx = sv->ctx;
  if (!sv->finished) return fail(ctx, SRCU_ERR_INVALID_ARGUMENT, "the stream is not finished");
  if (!out) return fail(ctx, SRCU_ERR_INVALID_ARGUMENT, "output is NULL");
  if (first > sv->voxels || count > sv->voxels - first)
    return fail(ctx, SRCU_ERR_INVALID_ARGUMENT, "voxels [%llu, %llu) are out of range (%llu voxels)",
                (unsigned long long)first, (unsigned long long)(first + count),
                (unsigned long long)sv->voxels);
  if (count == 0) return SRCU_OK;
  CU_TRY(cudaSetDevice(ctx->device));
  float *pos[3] = {out->x, out->y, out->z};
  TakeColumns t{};
  auto column = [&](void *dst, const DevBuf &src, uint32_t words) -> srcu_status {
    const uint32_t *from = static_cast<const uint32_t *>(src.p) + first * words;
    if (!out->on_device || !dst || !writable(ctx, dst))
      return copy_out(ctx, dst, from, count * words * 4, out->on_device);
    take_column(t, dst, from, words);
    return SRCU_OK;
  };
  for (int a = 0; a < 3; ++a) ST_TRY(column(pos[a], sv->opos[a], 1));
  for (uint32_t c = 3; c < sv->nc; ++c)
    if (out->attrs) ST_TRY(column(out->attrs[c - 3], sv->oattr[c], 2));
  ST_TRY(column(out->keys, sv->okeys, 6));
  ST_TRY(column(out->counts, sv->ocnt, 2));
  ST_TRY(take_columns(ctx, t, nullptr, count));
  CU_TRY(cudaStreamSynchronize(ctx->stream));
  return SRCU_OK;
}

void srcu_stream_voxel_destroy(srcu_stream_voxel *sv) {
  if (!sv) return;
  srcu_ctx *ctx = sv->ctx;
  cudaSetDevice(ctx->device);
  cudaStreamSynchronize(ctx->stream);
  if (!ctx->parked_stream) {  // kept for the context's next stream
    ctx->parked_stream = sv;
    return;
  }
  stream_voxel_free(sv);
}

}  // extern "C"

void stream_voxel_free(srcu_stream_voxel *sv) {
  if (!sv) return;
  sv_release(sv);
  if (sv->state_host) cudaFreeHost(sv->state_host);
  delete sv;
}
