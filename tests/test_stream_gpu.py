"""Bounded streaming voxel on the device (srcu_stream_voxel_*) vs the oracle.

Bar: the voxel key set, order and point counts are exact; positions are the
f32 of the FP64 mean (checked within 1e-5 of the leaf, and equal to the
oracle's f32 in all but rare FP64 rounding ties); FP64 attribute means
within 1e-12 relative.  The reference's own streaming tests
(streaming.rs:1098-1171) run through the Python mirror."""
import numpy as np
import pytest

import oracle
import spatialrust_b200 as sr
from spatialrust_b200 import _native, synthetic
from spatialrust_b200.streaming import (MemoryChunkSource, SpoolOptions, StreamingVoxelConfig,
                                        StreamingVoxelSource)

pytestmark = pytest.mark.gpu
F = np.float32


def xyz_cloud(points):
    b = sr.PointCloudBuilder.xyz()
    for p in points:
        b.push_point(p)
    return b.build()


def positions(src):
    out = []
    while (c := src.next_chunk()) is not None:
        out.extend(map(list, zip(c.field("x").tolist(), c.field("y").tolist(), c.field("z").tolist())))
    return out


def check_stream(ctx, x, y, z, attrs=(), leaf=0.1, chunk=100_000, device_run=0, f64=None):
    f64 = f64 if f64 is not None else [a.dtype == np.float64 for a in attrs]
    sv = _native.StreamVoxel(ctx, leaf, f64, device_run_points=device_run)
    for lo in range(0, len(x), chunk):
        sv.push(x[lo:lo + chunk], y[lo:lo + chunk], z[lo:lo + chunk], [a[lo:lo + chunk] for a in attrs])
    info = sv.finish()
    gx, gy, gz, ga, keys, counts = sv.fetch()
    sv.close()
    ref = oracle.stream_voxel(x, y, z, [np.asarray(a, np.float64) for a in attrs], leaf=leaf)
    assert info["voxels"] == len(ref.counts)
    assert np.array_equal(keys, ref.keys)
    assert np.array_equal(counts, ref.counts)
    pos = np.stack([gx, gy, gz], 1)
    assert np.max(np.abs(pos.astype(np.float64) - ref.pos)) <= 1e-5 * leaf + 1e-6 * np.abs(ref.pos).max()
    assert np.mean(pos == ref.pos) > 0.999
    if attrs:
        assert np.allclose(ga, ref.attrs, rtol=1e-12, atol=0)
    return info


# ---- the reference's streaming tests --------------------------------------

def test_output_identical_across_chunk_and_run_sizes(tmp_path):
    # streaming.rs:1098-1130
    pts = [[1.3, 0.0, 0.0], [0.1, 0.0, 0.0], [1.1, 0.0, 0.0], [0.2, 0.0, 0.0], [2.8, 0.0, 0.0]]
    sp = SpoolOptions(str(tmp_path), 16 * 1024)
    a = StreamingVoxelSource.try_build(MemoryChunkSource(xyz_cloud(pts), 1),
                                       StreamingVoxelConfig(1.0, 2, 8, sp))
    b = StreamingVoxelSource.try_build(MemoryChunkSource(xyz_cloud(pts), 4),
                                       StreamingVoxelConfig(1.0, 3, 8, sp))
    pa, pb = positions(a), positions(b)
    assert a.spool_bytes() > 0 and a.run_count() > 1
    assert pa == pb
    assert pa == np.array([[0.15, 0, 0], [1.2, 0, 0], [2.8, 0, 0]], F).tolist()


def test_attributes_averaged_across_runs(tmp_path):
    # streaming.rs:1132-1149
    b = sr.PointCloudBuilder(sr.StandardSchemas.point_xyzi())
    for p in ([0.1, 0.0, 0.0, 10.0], [0.2, 0.0, 0.0, 20.0], [1.1, 0.0, 0.0, 50.0]):
        b.push_point(p)
    src = StreamingVoxelSource.try_build(MemoryChunkSource(b.build(), 2),
                                         StreamingVoxelConfig(1.0, 1, 4,
                                                              SpoolOptions(str(tmp_path), 4096)))
    assert src.next_chunk().intensity().tolist() == [15.0, 50.0]


def test_spool_and_run_limits_fail_closed(tmp_path):
    # streaming.rs:1151-1171
    pts = xyz_cloud([[0.0, 0.0, 0.0], [1.0, 0.0, 0.0]])
    with pytest.raises(sr.InvalidArgument):
        StreamingVoxelSource.try_build(MemoryChunkSource(pts, 2),
                                       StreamingVoxelConfig(0.1, 2, 2, SpoolOptions(str(tmp_path), 8)))
    with pytest.raises(sr.InvalidArgument):
        StreamingVoxelSource.try_build(MemoryChunkSource(pts, 2),
                                       StreamingVoxelConfig(0.1, 1, 1, SpoolOptions(str(tmp_path), 4096)))


# ---- parity on larger streams ----------------------------------------------

def test_scan_stream_parity_with_runs_and_merge(cuda_ctx):
    c = synthetic.georef_scan(600_000, seed=51)
    # shuffled, so every voxel's points are spread over many device runs
    perm = np.random.default_rng(51).permutation(len(c.x))
    x, y, z, i = c.x[perm], c.y[perm], c.z[perm], c.intensity[perm]
    info = check_stream(cuda_ctx, x, y, z, [i], leaf=0.1, chunk=70_000, device_run=50_000)
    assert info["device_runs"] == 12 and info["partial_records"] > info["voxels"]


def test_long_voxels_in_runs_and_in_the_merge(cuda_ctx):
    # 3 voxels of ~100k points: long segments in every run, and (with 1000-point
    # device runs) more than 64 partial records per voxel in the merge
    rng = np.random.default_rng(7)
    p = rng.uniform(0, 3, (300_000, 3)).astype(F)
    p[:, 1:] = F(0.5)
    gps = 1e9 + rng.uniform(0, 100, 300_000)
    info = check_stream(cuda_ctx, p[:, 0], p[:, 1], p[:, 2], [gps], leaf=1.0, chunk=25_000,
                        device_run=1000)
    assert info["voxels"] == 3 and info["device_runs"] == 300


@pytest.mark.parametrize("f64", ["", "fd", "fdfdfd"])
def test_long_voxels_at_the_edges_of_a_block(cuda_ctx, f64):
    # one voxel per length: about the short limit (64), a block (256), the points a
    # block loads ahead (1024), and a block's rest after them
    sizes = [64, 65, 255, 256, 257, 767, 768, 769, 1023, 1024, 1025, 1279, 1280, 1281, 2047, 2049]
    rng = np.random.default_rng(23)
    x = rng.permutation(np.repeat(np.arange(len(sizes)), sizes)).astype(F) + F(0.25)
    y = rng.uniform(0, 0.9, len(x)).astype(F)
    z = rng.uniform(0, 0.9, len(x)).astype(F)
    attrs = [rng.uniform(1, 2, len(x)).astype(np.float64 if t == "d" else F) for t in f64]
    check_stream(cuda_ctx, x, y, z, attrs, leaf=1.0)


def test_non_finite_points_are_skipped_and_negative_keys(cuda_ctx):
    rng = np.random.default_rng(8)
    p = rng.normal(0, 5, (50_000, 3)).astype(F)
    p[::7, 0] = np.nan
    p[::11, 2] = np.inf
    p[::13, 1] = -np.inf
    info = check_stream(cuda_ctx, p[:, 0], p[:, 1], p[:, 2], leaf=0.25, chunk=9_999, device_run=20_000)
    finite = np.all(np.isfinite(p), axis=1).sum()
    assert info["finite_points"] == finite and info["points"] == 50_000


@pytest.mark.parametrize("f64", [False, True])
@pytest.mark.parametrize("device_run", [0, 1, 2, 5])
def test_non_finite_attributes(cuda_ctx, device_run, f64):
    # a voxel per sequence, in one run and over merged runs: an infinity that others
    # follow ends as NaN, as the compensated sum of the whole stream does, a last one as
    # itself.  Sums of small integers: nothing rounds but the mean, one division.
    inf, nan = np.inf, np.nan
    sequences = [[inf, 1.0], [1.0, inf], [inf, 1.0, 2.0], [1.0, inf, 2.0], [1.0, 2.0, -inf], [-inf],
                 [-inf, 3.0], [inf, -inf], [inf, inf], [nan, 1.0], [1.0, nan], [-0.0], [-0.0, -0.0],
                 [-0.0, inf], [4.0, 5.0, 6.0], [inf] + [1.0] * 80]
    x = np.concatenate([[F(v)] * len(s) for v, s in enumerate(sequences)]).astype(F)
    values = np.concatenate(sequences).astype(np.float64 if f64 else F)
    zero = np.zeros_like(x)
    sv = _native.StreamVoxel(cuda_ctx, 1.0, [f64], device_run_points=device_run)
    sv.push(x, zero, zero, [values])
    assert sv.finish()["voxels"] == len(sequences)
    attrs, counts = sv.fetch()[3], sv.fetch()[5]
    sv.close()
    ref = oracle.stream_voxel(x, zero, zero, [values.astype(np.float64)], leaf=1.0)
    assert np.array_equal(counts, ref.counts)
    assert np.array_equal(attrs, ref.attrs, equal_nan=True)


def test_all_points_non_finite_or_empty(cuda_ctx):
    sv = _native.StreamVoxel(cuda_ctx, 1.0)
    sv.push(np.full(10, np.nan, F), np.zeros(10, F), np.zeros(10, F))
    assert sv.finish()["voxels"] == 0
    sv.close()
    sv = _native.StreamVoxel(cuda_ctx, 1.0)
    assert sv.finish()["voxels"] == 0
    sv.close()


def test_device_chunks_and_f32_attributes(cuda_ctx):
    import torch
    c = synthetic.shapes_scene(200_000, seed=12)
    inten = np.random.default_rng(12).random(200_000).astype(F)
    host = _native.StreamVoxel(cuda_ctx, 0.05, [False])
    dev = _native.StreamVoxel(cuda_ctx, 0.05, [False])
    for lo in range(0, 200_000, 64_000):
        sl = slice(lo, lo + 64_000)
        host.push(c.x[sl], c.y[sl], c.z[sl], [inten[sl]])
        dev.push(*[torch.from_numpy(np.ascontiguousarray(a[sl])).cuda() for a in (c.x, c.y, c.z)],
                 [torch.from_numpy(inten[sl]).cuda()])
    assert host.finish()["voxels"] == dev.finish()["voxels"]
    for a, b in zip(host.fetch(), dev.fetch()):
        assert np.array_equal(a, b)
    host.close()
    dev.close()


def test_key_range_error_and_bad_arguments(cuda_ctx):
    sv = _native.StreamVoxel(cuda_ctx, 1e-12)
    sv.push(np.array([1e30], F), np.zeros(1, F), np.zeros(1, F))
    with pytest.raises(sr.InvalidArgument, match="64-bit range"):
        sv.finish()
    sv.close()
    for leaf in (0.0, -1.0, float("nan"), float("inf")):
        with pytest.raises(sr.InvalidArgument):
            _native.StreamVoxel(cuda_ctx, leaf)
    sv = _native.StreamVoxel(cuda_ctx, 1.0, [False])
    with pytest.raises(sr.InvalidArgument):
        sv.push(np.zeros(3, F), np.zeros(3, F), np.zeros(3, F))
    with pytest.raises(sr.BufferLengthMismatch):
        sv.push(np.zeros(3, F), np.zeros(2, F), np.zeros(3, F), [np.zeros(3, F)])
    sv.close()


@pytest.mark.parametrize("f64", ["", "d", "f", "dfd", "ddff", "fdfdfdfdf", "ddddddddd"])
@pytest.mark.parametrize("n,device_run", [(1, 0), (1023, 0), (1025, 1025), (5000, 700)])
def test_record_layouts(cuda_ctx, f64, n, device_run):
    """Every mix of attribute types is packed into point records and back: one
    run straight into the outputs, exactly one full run, and merged runs."""
    rng = np.random.default_rng(n + len(f64))
    p = rng.uniform(-2, 2, (3, n)).astype(F)
    attrs = [rng.normal(0, 3, n).astype(np.float64 if t == "d" else F) for t in f64]
    info = check_stream(cuda_ctx, *p, attrs, leaf=0.4, chunk=333, device_run=device_run)
    assert info["device_runs"] == (1 if device_run == 0 else -(-n // device_run))


def test_device_columns_off_their_alignment(cuda_ctx):
    """FP64 device columns that start off an 8-byte boundary are staged."""
    import ctypes
    import torch
    n = 4000
    rng = np.random.default_rng(3)
    p = rng.uniform(0, 5, (3, n)).astype(F)
    g = rng.normal(0, 1, n)
    raw = torch.zeros(8 * n + 4, dtype=torch.uint8, device="cuda")
    raw[4:] = torch.from_numpy(g.view(np.uint8)).cuda()
    cols = [torch.from_numpy(a).cuda() for a in p]
    out = []
    aligned = torch.from_numpy(g).cuda()
    for address in (raw.data_ptr() + 4, aligned.data_ptr()):
        sv = _native.StreamVoxel(cuda_ctx, 0.5, [True])
        attrs = (ctypes.c_void_p * 1)(address)
        cloud = _native.SrcuCloud(*[c.data_ptr() for c in cols],
                                  ctypes.cast(attrs, ctypes.c_void_p), 1, 1, n)
        cuda_ctx._check(cuda_ctx._lib.srcu_stream_voxel_push(sv._h, ctypes.byref(cloud)))
        sv.finish()
        out.append(sv.fetch())
        sv.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("offset", [0, 1, 2, 4])
def test_fetch_to_device_at_any_alignment(cuda_ctx, offset):
    """Device columns that start off a word or a 16-byte boundary hold the bytes that
    host columns hold, with nothing written past them."""
    import ctypes
    import torch
    rng = np.random.default_rng(5)
    sv = _native.StreamVoxel(cuda_ctx, 0.5, [True])
    sv.push(*rng.uniform(0, 9, (3, 3000)).astype(F), [rng.normal(0, 1, 3000)])
    sv.finish()
    x, y, z, a, keys, counts = sv.fetch()
    want = [x, y, z, a[:, 0], keys, counts]
    bufs = [torch.full((w.nbytes + 16,), 0xA5, dtype=torch.uint8, device="cuda") for w in want]
    at = [b.data_ptr() + offset for b in bufs]
    attrs = (ctypes.c_void_p * 1)(at[3])
    out = _native.SrcuStreamVoxelOut(*at[:3], ctypes.cast(attrs, ctypes.c_void_p), at[4], at[5], 1)
    cuda_ctx._check(cuda_ctx._lib.srcu_stream_voxel_fetch(sv._h, 0, len(x), ctypes.byref(out)))
    sv.close()
    for b, w in zip(bufs, want):
        w = np.ascontiguousarray(w).reshape(-1).view(np.uint8)
        got = b.cpu().numpy()
        assert np.array_equal(got[offset:offset + len(w)], w)
        assert np.all(got[:offset] == 0xA5) and np.all(got[offset + len(w):] == 0xA5)


def test_chunks_outside_device_memory_are_staged(cuda_ctx):
    # pinned host memory marked as device memory: no kernel reads the caller's columns,
    # they are copied into staging columns, which the context's byte count shows
    import ctypes
    import torch
    n = 5000
    c = synthetic.shapes_scene(n, seed=4)
    cols = [torch.from_numpy(np.ascontiguousarray(a, F)) for a in (c.x, c.y, c.z)]
    got, staged = {}, {}
    for name, held in (("device", [t.cuda() for t in cols]), ("pinned", [t.pin_memory() for t in cols])):
        torch.cuda.synchronize()
        ctx = _native.Context(0)
        sv = _native.StreamVoxel(ctx, 0.05, device_run_points=n)
        before = ctx.device_bytes()
        chunk = _native.SrcuCloud(*[t.data_ptr() for t in held], None, 0, 1, n)
        ctx._check(ctx._lib.srcu_stream_voxel_push(sv._h, ctypes.byref(chunk)))
        # the chunk fills the run, whose reduction allocates the same for both
        staged[name] = ctx.device_bytes() - before
        sv.finish()
        got[name] = sv.fetch()
        sv.close()
        ctx.close()
    assert staged["pinned"] - staged["device"] >= 3 * 4 * n
    for a, b in zip(got["device"], got["pinned"]):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("device_run", [0, 1, 64, 1000, 65_537])
def test_host_and_device_chunks_in_turn(cuda_ctx, device_run):
    """Chunks gathered in the staging columns, chunks read in place between them, and
    the ends of runs and of the staging columns: as if pushed at once, and twice over
    with the buffers of the first stream, whose columns had other types."""
    import torch
    rng = np.random.default_rng(device_run)
    sizes = [1, 3, 0, 63, 64, 65, 2, 700, 1, 300] if device_run in (1, 64) else \
        [1, 3, 0, 65_536, 1, 65_535, 2, 70_000, 700, 1]
    n = sum(sizes)
    p = rng.uniform(0, 12, (n, 3)).astype(F)
    extra = [rng.random(n), rng.random(n)]
    for f64 in ([True, False], [False, True]):
        attrs = [a.astype(np.float64 if f else F) for a, f in zip(extra, f64)]
        cols = [np.ascontiguousarray(p[:, k]) for k in range(3)] + attrs
        sv = _native.StreamVoxel(cuda_ctx, 1.0, f64, device_run_points=device_run)
        lo = 0
        for i, m in enumerate(sizes):
            part = [c[lo:lo + m] for c in cols]
            if i % 3 == 2:
                part = [torch.from_numpy(np.ascontiguousarray(c)).cuda() for c in part]
                torch.cuda.synchronize()
            sv.push(*part[:3], part[3:])
            lo += m
        assert sv.finish()["points"] == n
        got = sv.fetch()
        sv.close()
        ref = oracle.stream_voxel(*cols[:3], [a.astype(np.float64) for a in attrs], leaf=1.0)
        assert np.array_equal(got[4], ref.keys) and np.array_equal(got[5], ref.counts)
        assert np.allclose(got[3], ref.attrs, rtol=1e-12, atol=0)
