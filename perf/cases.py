"""Performance cases of the uniform-grid path, through the calls a program makes.

listed() names the cases, draw() makes more of the same ranges, prepare() builds
what a program holds before the call, run() is one pass, work() what a pass
cannot do without, exact() the same outputs in 64 bits from plain torch.

Kinds of case, with what each stands for:

    host     srcu_voxel_centroid on host columns, in and out: the drop-in call of
             a Gpu(Cuda) voxel filter
    chain    one device-resident cloud: voxel centroids, then radius normals on
             them, results taken into the caller's device columns (a frame or
             one scan)
    batch    many uneven clouds in one chain (map tiles, recorded frames), results
             taken as above
    normals  radius normals of a raw cloud, device in and out
    cluster  Euclidean cluster roots of a raw cloud
    plane    GICP plane covariances of a raw cloud
    ransac   RANSAC plane segmentation of a raw cloud
    las      LAS point records decoded to columns
    stream   bounded streaming voxel: pushed chunks, finish, fetch

A result whose length depends on the input goes into the caller's columns of
the input's length, zero past its end.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from spatialrust_b200 import _native, las

DEV = "cuda"
VIEWPOINT = (0.0, 0.0, 100.0)  # chains on scans: above the scan, as an airborne sensor
RUN_POINTS = 1 << 20           # run length of the streaming cases' spool accounting


def listed():
    return [
        # the drop-in call on a small crop: launches, copies and waits
        dict(name="host_filter_20k", kind="host", mode="average", n=20_000, attrs=1, leaf=0.2),
        # the drop-in call on a cloud of bare positions (first-seen voxel order)
        dict(name="host_filter_xyz_300k", kind="host", mode="xyz", n=300_001, attrs=0, leaf=0.1),
        # one spinning-LiDAR frame (64 beams x 2048 azimuths), the serving parameters
        dict(name="frame_131k", kind="chain", scene="lidar", beams=64, azimuths=2048, attrs=1,
             leaf=0.2, radius=0.6),
        # the headline scan: fine voxels, nearly one point each
        dict(name="scan_2M_fine", kind="chain", scene="scan", n=2_000_000, attrs=1, leaf=0.1,
             radius=0.5),
        # the same scan at coarse voxels, with four attribute columns
        dict(name="scan_2M_coarse", kind="chain", scene="scan", n=2_000_000, attrs=4, leaf=0.5,
             radius=0.5),
        # uneven map tiles in one chain, 10k to 1M points each
        dict(name="batch_64", kind="batch", clouds=64, lo=10_000, hi=1_000_000),
        # dense surfaces: hundreds of neighbours per point
        dict(name="normals_5M", kind="normals", n=5_000_000, radius=0.3, include_self=False),
        # object clusters of a raw scan
        dict(name="cluster_2M", kind="cluster", n=2_000_000, tolerance=0.3),
        # registration covariances of a raw scan
        dict(name="plane_cov_2M", kind="plane", n=1_999_999, radius=0.3),
        # ground plane of a scan, the default 1000 hypotheses
        dict(name="ransac_460k", kind="ransac", n=460_000, hypotheses=1000, threshold=0.01),
        # ingest: LAS 1.4 format-1 records (28 bytes)
        dict(name="las_8M", kind="las", n=8_000_001, format=1),
        # a map larger than one device run, pushed in chunks
        dict(name="stream_8M", kind="stream", n=8_000_003, chunk=1_000_000, leaf=0.1),
    ]


def _size(rng, lo, hi):
    """A size spread over the logarithm of [lo, hi], odd ones among them."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "chain", "chain", "chain", "batch", "normals", "cluster", "plane",
                       "ransac", "las", "stream"])
    if kind == "host":
        mode = rng.choice(["average", "average", "xyz", "first", "approximate"])
        return dict(kind=kind, mode=mode, n=_size(rng, 2_000, 500_000),
                    attrs=0 if mode == "xyz" else rng.choice([1, 3, 4]),
                    leaf=round(rng.uniform(0.05, 0.5), 3))
    if kind == "chain":
        attrs = rng.choice([0, 1, 1, 3, 4])
        if rng.random() < 0.4:
            leaf = round(rng.uniform(0.1, 0.4), 3)
            return dict(kind=kind, scene="lidar", beams=rng.choice([16, 32, 64, 128]),
                        azimuths=rng.randint(512, 2048), attrs=attrs, leaf=leaf,
                        radius=round(3.0 * leaf, 3))
        return dict(kind=kind, scene="scan", n=_size(rng, 50_000, 4_000_000), attrs=attrs,
                    leaf=round(rng.uniform(0.05, 0.5), 3), radius=0.5)
    if kind == "batch":
        lo = _size(rng, 2_000, 20_000)
        return dict(kind=kind, clouds=rng.randint(2, 64), lo=lo, hi=lo * rng.randint(2, 30))
    if kind == "normals":
        return dict(kind=kind, n=_size(rng, 50_000, 4_000_000), radius=round(rng.uniform(0.1, 0.3), 3),
                    include_self=rng.random() < 0.5)
    if kind == "cluster":
        return dict(kind=kind, n=_size(rng, 20_000, 3_000_000),
                    tolerance=round(rng.uniform(0.05, 0.35), 3))
    if kind == "plane":
        return dict(kind=kind, n=_size(rng, 20_000, 3_000_000), radius=round(rng.uniform(0.2, 0.4), 3))
    if kind == "ransac":
        return dict(kind=kind, n=_size(rng, 5_000, 1_000_000), hypotheses=rng.randint(100, 2000),
                    threshold=rng.choice([0.01, 0.02, 0.05]))
    if kind == "las":
        return dict(kind=kind, n=_size(rng, 20_000, 8_000_000), format=rng.choice([0, 1, 3, 6, 7]))
    return dict(kind=kind, n=_size(rng, 100_000, 8_000_000), chunk=_size(rng, 65_536, 1_000_000),
                leaf=round(rng.uniform(0.05, 0.5), 3))


# ---- inputs, made on the GPU from the seed -----------------------------------

def _rng(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _uniform(g, shape, lo=0.0, hi=1.0):
    return torch.rand(shape, generator=g, device=DEV, dtype=torch.float64) * (hi - lo) + lo


def _normal(g, shape, sigma=1.0):
    return torch.randn(shape, generator=g, device=DEV, dtype=torch.float64) * sigma


def _scan(g, n, square=200.0, boxes=200):
    """Ground (60%), faces of boxes standing on it (30%) and clutter (10%), in
    random order: (n, 3) float64 about the scan's own origin."""
    n_ground, n_box = int(round(n * 0.6)), int(round(n * 0.3))
    pts = _uniform(g, (n, 3))
    pts[:, :2] *= square
    pts[:n_ground, 2] = _normal(g, (n_ground,), 0.02)
    pts[n_ground + n_box:, 2] *= 20.0
    size = _uniform(g, (boxes, 3), 0.5, 8.0)
    low = torch.cat([_uniform(g, (boxes, 2), 0.0, square), torch.zeros((boxes, 1), device=DEV,
                                                                       dtype=torch.float64)], 1)
    sx, sy, sz = size.T
    area = torch.stack([sx * sy, sx * sz, sx * sz, sy * sz, sy * sz], 1).reshape(-1)  # no bottom
    pick = torch.multinomial(area, n_box, replacement=True, generator=g)
    box, face = pick // 5, pick % 5
    u = pts[n_ground:n_ground + n_box]
    u[:, :2] = _uniform(g, (n_box, 2))
    for f, axis, side in ((0, 2, 1.0), (1, 1, 0.0), (2, 1, 1.0), (3, 0, 0.0), (4, 0, 1.0)):
        u[:, axis] = torch.where(face == f, side, u[:, axis])
    u.mul_(size[box]).add_(low[box])
    return pts[torch.randperm(n, generator=g, device=DEV)]


def _shapes(g, n, extent=100.0, noise=0.005):
    """Spheres (40%), planar patches (40%) and cylinders (20%) with surface noise."""
    n_sph, n_pl = int(round(n * 0.4)), int(round(n * 0.4))
    n_cyl = n - n_sph - n_pl

    def rotations(k):
        return torch.linalg.qr(_normal(g, (k, 3, 3)))[0]

    rad, cen = _uniform(g, (50,), 1.0, 5.0), _uniform(g, (50, 3), 8.0, extent - 8.0)
    which = torch.multinomial(rad ** 2, n_sph, replacement=True, generator=g)
    d = torch.nn.functional.normalize(_normal(g, (n_sph, 3)), dim=1)
    sph = cen[which] + d * (rad[which] + _normal(g, (n_sph,), noise))[:, None]
    rot, cen = rotations(30), _uniform(g, (30, 3), 8.0, extent - 8.0)
    which = torch.randint(0, 30, (n_pl,), generator=g, device=DEV)
    local = torch.cat([_uniform(g, (n_pl, 2), -5.0, 5.0), _normal(g, (n_pl, 1), noise)], 1)
    pl = cen[which] + torch.einsum("nij,nj->ni", rot[which], local)
    rot, cen, rad = rotations(20), _uniform(g, (20, 3), 8.0, extent - 8.0), _uniform(g, (20,), 0.2, 1.0)
    which = torch.multinomial(rad, n_cyl, replacement=True, generator=g)
    th, h = _uniform(g, (n_cyl,), 0.0, 2 * math.pi), _uniform(g, (n_cyl,), -2.5, 2.5)
    rr = rad[which] + _normal(g, (n_cyl,), noise)
    local = torch.stack([rr * th.cos(), rr * th.sin(), h], 1)
    cyl = cen[which] + torch.einsum("nij,nj->ni", rot[which], local)
    return torch.cat([sph, pl, cyl])[torch.randperm(n, generator=g, device=DEV)]


def _lidar(g, beams, azimuths, max_range=120.0):
    """One spinning-LiDAR frame in the sensor frame, beam by beam: first hits of
    the rays on the ground (1.8 m below) and on 100 boxes, with range noise."""
    size = _uniform(g, (100, 3), 0.5, 8.0)
    low = torch.cat([_uniform(g, (100, 2), -120.0, 120.0),
                     torch.full((100, 1), -1.8, device=DEV, dtype=torch.float64)], 1)
    near = (low[:, :2] < 1.0).all(1) & (low[:, :2] + size[:, :2] > -1.0).all(1)
    low, size = low[~near], size[~near]  # no box over the sensor
    el = torch.linspace(math.radians(-25.0), math.radians(15.0), beams, device=DEV,
                        dtype=torch.float64)[:, None]
    az = torch.arange(azimuths, device=DEV, dtype=torch.float64)[None] * (2 * math.pi / azimuths)
    d = torch.stack([el.cos() * az.cos(), el.cos() * az.sin(), el.sin().expand(beams, azimuths)],
                    -1).reshape(-1, 3)
    t = torch.where(d[:, 2] < -1e-9, -1.8 / d[:, 2], max_range).clamp(max=max_range)
    inv = 1.0 / d
    for a, b in zip(low, low + size):
        t1, t2 = a * inv, b * inv
        tn, tf = torch.minimum(t1, t2).amax(1), torch.maximum(t1, t2).amin(1)
        t = torch.where((tn <= tf) & (tn > 0.0) & (tn < t), tn, t)
    r = (t + _normal(g, t.shape, 0.02)).clamp(1e-3, max_range)
    return d * r[:, None]


def _columns(xyz):
    return [xyz[:, a].to(torch.float32).contiguous() for a in range(3)]


def _attributes(g, n, count):
    return [torch.rand(n, generator=g, device=DEV) for _ in range(count)]


def _batch_sizes(case):
    """Points and leaf of every cloud of a batch: a property of the case."""
    r = np.random.default_rng([case["clouds"], case["lo"], case["hi"]])
    sizes = np.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"]), case["clouds"]))
    return sizes.astype(np.int64).tolist(), r.choice([0.05, 0.1, 0.2], case["clouds"]).tolist()


def _las_layout(fmt):
    """(record length, classification, GPS time and RGB offsets) of a record format."""
    length, gps, rgb = las.LAS_LAYOUTS[fmt]
    return length, (16 if fmt >= 6 else 15), gps, rgb


LAS_SCALE, LAS_ORIGIN = 0.001, (450_000.0, 3_900_000.0, 50.0)


def _las_fields(case, seed):
    g, n = _rng(seed), case["n"]
    raw = (_scan(g, n) / LAS_SCALE).round().to(torch.int32)  # stored about the origin
    f = dict(xyz=raw, intensity=torch.randint(0, 32768, (n,), generator=g, device=DEV),
             cls=torch.randint(0, 32, (n,), generator=g, device=DEV),
             gps=1.4e9 + torch.arange(n, device=DEV, dtype=torch.float64) * 1e-5,
             rgb=torch.randint(0, 32768, (n, 3), generator=g, device=DEV))
    return f


def _inputs(case, seed):
    """The case's input columns: positions, then attributes."""
    g, kind = _rng(seed), case["kind"]
    if kind == "chain":
        xyz = (_lidar(g, case["beams"], case["azimuths"]) if case["scene"] == "lidar"
               else _scan(g, case["n"]))
        return _columns(xyz) + _attributes(g, xyz.shape[0], case["attrs"])
    if kind == "batch":
        xyz = torch.cat([_scan(g, n) for n in _batch_sizes(case)[0]])
        return _columns(xyz) + _attributes(g, xyz.shape[0], 1)
    if kind == "normals":
        return _columns(_shapes(g, case["n"]))
    if kind == "stream":
        cols = _columns(_scan(g, case["n"])) + _attributes(g, case["n"], 1)
        return cols + [1.4e9 + torch.arange(case["n"], device=DEV, dtype=torch.float64) * 1e-5]
    return _columns(_scan(g, case["n"])) + _attributes(g, case["n"], case.get("attrs", 0))


# ---- one pass -----------------------------------------------------------------

def _voxel_out(columns, counts, on_device, keep):
    attrs = keep.add((ctypes.c_void_p * max(1, len(columns) - 3))(*[_native._addr(c)
                                                                   for c in columns[3:]]))
    return _native.SrcuVoxelOut(*[_native._addr(c) for c in columns[:3]],
                                ctypes.cast(attrs, ctypes.c_void_p), 0, _native._addr(counts),
                                on_device)


def _fetch(s):
    """The chain's results into the caller's device columns."""
    ctx, voxels, stats = s["ctx"], ctypes.c_uint64(0), _native.SrcuNormalStats()
    ctx._check(_native.load().srcu_frame_fetch(ctx.handle, ctypes.byref(s["vout"]),
                                               ctypes.byref(s["nout"]), ctypes.byref(voxels),
                                               ctypes.byref(stats)))
    return dict(columns=s["columns"], counts=s["counts"], normals=s["normals"][:3],
                curvature=s["normals"][3], neighbors=s["neighbors"], voxels=voxels.value,
                valid=stats.valid_count)


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    s["ctx"] = _native.shared_context()
    if kind == "las":
        f, n = _las_fields(case, seed), case["n"]
        length, cls, gps, rgb = _las_layout(case["format"])
        rec = torch.zeros((n, length), dtype=torch.uint8, device=DEV)
        rec[:, 0:12] = f["xyz"].contiguous().view(torch.uint8).reshape(n, 12)
        rec[:, 12:14] = f["intensity"].to(torch.int16).view(torch.uint8).reshape(n, 2)
        rec[:, cls] = f["cls"].to(torch.uint8)
        if gps is not None:
            rec[:, gps:gps + 8] = f["gps"].view(torch.uint8).reshape(n, 8)
        if rgb is not None:
            rec[:, rgb:rgb + 6] = f["rgb"].to(torch.int16).contiguous().view(torch.uint8).reshape(n, 6)
        s["records"] = rec.reshape(-1)
        s["header"] = las.LasHeader((1, 4), 375, 375, case["format"], length, n, (LAS_SCALE,) * 3,
                                    LAS_ORIGIN, (0.0,) * 3, (0.0,) * 3, False)
        return s
    cols = s["cols"] = _inputs(case, seed)
    n = cols[0].shape[0]
    s["keep"] = _native._Keep()
    if kind == "host":
        cols = s["cols"] = [c.cpu().numpy() for c in cols]
        s["columns"] = [np.zeros_like(c) for c in cols]
        s["counts"] = np.zeros(n, np.int32)
        s["vout"] = _voxel_out(s["columns"], s["counts"], 0, s["keep"])
        s["params"] = _native._voxel_params(case["leaf"], None, case["mode"] == "approximate",
                                            case["mode"] in ("first", "approximate"),
                                            case["mode"] == "xyz")
    if kind != "stream":
        s["cloud"] = _native.make_cloud(*cols[:3], cols[3:], s["keep"])
    if kind in ("chain", "batch"):
        s["columns"] = [torch.zeros_like(c) for c in cols]
        s["normals"] = [torch.zeros_like(cols[0]) for _ in range(4)]
        s["counts"], s["neighbors"] = (torch.zeros(n, dtype=torch.int32, device=DEV)
                                       for _ in range(2))
        s["vout"] = _voxel_out(s["columns"], s["counts"], 1, s["keep"])
        s["nout"] = _native.SrcuNormalOut(*[c.data_ptr() for c in s["normals"]],
                                          s["neighbors"].data_ptr(), 1)
    if kind == "batch":
        sizes, s["leaves"] = _batch_sizes(case)
        s["offsets"] = np.concatenate([[0], np.cumsum(sizes)]).tolist()
        s["radii"] = [5.0 * v for v in s["leaves"]]
    if kind in ("normals", "plane"):
        s["out"] = [torch.empty(n, device=DEV) for _ in range(4)]
        s["counts"] = torch.empty(n, dtype=torch.int32, device=DEV)
        s["cov"] = torch.empty((n, 6), device=DEV)
    if kind == "stream":
        s["pos"] = [torch.zeros(n, device=DEV) for _ in range(3)]
        s["mean"] = [torch.zeros(n, dtype=torch.float64, device=DEV) for _ in range(2)]
        s["keys"] = torch.zeros((n, 3), dtype=torch.int64, device=DEV)
        s["counts"] = torch.zeros(n, dtype=torch.int64, device=DEV)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    ctx = s["ctx"]
    if kind == "host":
        voxels = ctypes.c_uint64(0)
        ctx._check(_native.load().srcu_voxel_centroid(
            ctx.handle, ctypes.byref(s["cloud"]), ctypes.byref(s["params"]), ctypes.byref(s["vout"]),
            ctypes.byref(voxels)))
        return dict(columns=s["columns"], counts=s["counts"], voxels=voxels.value)
    if kind == "chain":
        view = (0.0, 0.0, 0.0) if case["scene"] == "lidar" else VIEWPOINT
        ctx.voxel_normals_enqueue(s["cloud"], case["leaf"], None, case["radius"], 3, view,
                                  count_shell=False)
        return _fetch(s)
    if kind == "batch":
        count = case["clouds"]
        ctx.batch_voxel_normals_enqueue(s["cloud"], s["offsets"], s["leaves"], s["radii"], 3,
                                        [VIEWPOINT] * count, count_shell=False)
        return dict(_fetch(s), offsets=ctx.batch_voxel_offsets())
    if kind == "normals":
        out = _native.SrcuNormalOut(*[o.data_ptr() for o in s["out"]], s["counts"].data_ptr(), 1)
        prm = _native._normal_params(case["radius"], 3, VIEWPOINT, case["include_self"])
        stats = _native.SrcuNormalStats()
        ctx._check(_native.load().srcu_radius_normals(ctx.handle, ctypes.byref(s["cloud"]),
                                                      ctypes.byref(prm), ctypes.byref(out),
                                                      ctypes.byref(stats)))
        return dict(normals=s["out"][:3], curvature=s["out"][3], counts=s["counts"],
                    valid=stats.valid_count, shell=stats.shell_points)
    if kind == "cluster":
        return ctx.euclidean_cluster_roots(*s["cols"], case["tolerance"])
    if kind == "plane":
        stats = _native.SrcuNormalStats()
        ctx._check(_native.load().srcu_plane_covariances(
            ctx.handle, ctypes.byref(s["cloud"]), ctypes.c_float(case["radius"]),
            ctypes.c_float(1e-3), s["cov"].data_ptr(), ctypes.byref(stats)))
        return dict(cov=s["cov"], valid=stats.valid_count)
    if kind == "ransac":
        info, mask = ctx.ransac_plane_segment(*s["cols"], case["threshold"], case["hypotheses"], 3, 42)
        return dict(info, mask=mask)
    if kind == "las":
        return las.decode_records(s["records"], s["header"], LAS_ORIGIN)
    sv = _native.StreamVoxel(ctx, case["leaf"], [False, True], RUN_POINTS)
    n, step = case["n"], case["chunk"]
    for lo in range(0, n, step):
        x, y, z, intensity, gps = (c[lo:lo + step] for c in s["cols"])
        sv.push(x, y, z, [intensity, gps])
    info = sv.finish()
    v = info["voxels"]
    attrs = (ctypes.c_void_p * 2)(*[m.data_ptr() for m in s["mean"]])
    out = _native.SrcuStreamVoxelOut(*[p.data_ptr() for p in s["pos"]],
                                     ctypes.cast(attrs, ctypes.c_void_p), s["keys"].data_ptr(),
                                     s["counts"].data_ptr(), 1)
    ctx._check(_native.load().srcu_stream_voxel_fetch(sv._h, 0, v, ctypes.byref(out)))
    sv.close()
    return dict(pos=s["pos"], mean=s["mean"], keys=s["keys"], counts=s["counts"], voxels=v,
                runs=info["runs"], finite=info["finite_points"])


# ---- what a pass cannot do without ----------------------------------------------

def work(case):
    """Input columns read once, result rows written once.  The number of voxels
    depends on the input: a voxel per point is counted for fine leaves on these
    scenes, and the cells of the ground alone for coarse ones."""
    kind = case["kind"]
    if kind == "batch":
        sizes, leaves = _batch_sizes(case)
        n = sum(sizes)
        return dict(bytes=16.0 * n + 40.0 * sum(map(_voxels, sizes, leaves)), flops=0.0)
    n = case["beams"] * case["azimuths"] if case.get("scene") == "lidar" else case["n"]
    if kind == "host":
        row = 12.0 + 4.0 * case["attrs"]
        return dict(bytes=row * n + (row + 4.0) * _voxels(n, case["leaf"]), flops=0.0)
    if kind == "chain":
        row = 12.0 + 4.0 * case["attrs"]
        v = _voxels(n, case["leaf"]) if case["scene"] == "scan" else 0.5 * n
        return dict(bytes=row * n + (row + 24.0) * v, flops=0.0)
    if kind == "normals":
        return dict(bytes=32.0 * n, flops=0.0)
    if kind == "cluster":
        return dict(bytes=16.0 * n, flops=0.0)
    if kind == "plane":
        return dict(bytes=36.0 * n, flops=0.0)
    if kind == "ransac":  # an evaluation is three products, three sums and a comparison
        return dict(bytes=13.0 * n, flops=7.0 * n * case["hypotheses"])
    if kind == "las":
        length, _, gps, rgb = _las_layout(case["format"])
        return dict(bytes=n * (length + 17.0 + (8.0 if gps is not None else 0.0)
                               + (6.0 if rgb is not None else 0.0)), flops=0.0)
    return dict(bytes=24.0 * n + 60.0 * _voxels(n, case["leaf"]), flops=0.0)


def _voxels(n, leaf, square=200.0):
    """Voxels of a scan of n points: the ground's cells hit, and the rest apart."""
    cells = (square / leaf) ** 2
    return cells * -math.expm1(-0.6 * n / cells) + 0.3 * n * min(1.0, leaf * 4.0) + 0.1 * n


# ---- the same outputs in 64 bits ---------------------------------------------------

def _voxel_groups(cols, leaf):
    """(group of each point, voxels, points per voxel) in ascending key order,
    with the reference's float32 key of a min-corner origin."""
    inv = torch.tensor(1.0, device=DEV) / torch.tensor(leaf, device=DEV, dtype=torch.float32)
    k = [((c - c.min()) * inv).to(torch.int64) for c in cols[:3]]
    _, group, count = torch.unique(_pack(k), return_inverse=True, return_counts=True)
    return group, count.shape[0], count


def _pack(k):
    d1, d2 = int(k[1].max()) + 3, int(k[2].max()) + 3
    return (k[0] * d1 + k[1]) * d2 + k[2]


def _first(group, voxels):
    at = torch.arange(group.shape[0], device=DEV)
    return torch.full((voxels,), group.shape[0], device=DEV).scatter_reduce(0, group, at, "amin")


def _means(cols, group, voxels, count):
    return [torch.zeros(voxels, device=DEV, dtype=torch.float64).index_add_(0, group, c.double())
            / count for c in cols]


def _moments(cols, radius):
    """Neighbours (the query among them) by the float32 predicate, and their
    float64 moments about the query: count, sums, sums of products."""
    p = torch.stack(cols, 1)
    n = p.shape[0]
    cell = ((p.double() - p.double().amin(0)) / (radius * (1 + 1e-5))).floor().to(torch.int64) + 1
    d1, d2 = int(cell[:, 1].max()) + 2, int(cell[:, 2].max()) + 2
    key, order = torch.sort((cell[:, 0] * d1 + cell[:, 1]) * d2 + cell[:, 2], stable=True)
    q = p[order].contiguous()
    r = torch.tensor(radius, device=DEV, dtype=torch.float32)
    out = torch.zeros((n, 10), device=DEV, dtype=torch.float64)
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            mid = key + (dx * d1 + dy) * d2
            lo = torch.searchsorted(key, mid - 1)
            length = torch.searchsorted(key, mid + 1, right=True) - lo
            at = 0
            while at < n:
                rows = min(n - at, 1 << 18)
                while rows > 256 and rows * int(length[at:at + rows].max()) > 1 << 25:
                    rows //= 2
                ln = length[at:at + rows, None]
                step = torch.arange(int(ln.max()), device=DEV)[None]
                if step.shape[1]:
                    c = q[(lo[at:at + rows, None] + step).clamp(max=n - 1)]
                    d = c - q[at:at + rows, None]
                    sq = d * d
                    hit = ((sq[..., 0] + sq[..., 1]) + sq[..., 2] <= r * r) & (step < ln)
                    d = torch.where(hit[..., None], c.double() - q[at:at + rows, None].double(), 0.0)
                    o = out[at:at + rows]
                    o[:, 0] += hit.sum(1)
                    o[:, 1:4] += d.sum(1)
                    o[:, 4:7] += (d * d).sum(1)
                    for k, (a, b) in enumerate(((0, 1), (0, 2), (1, 2))):
                        o[:, 7 + k] += (d[..., a] * d[..., b]).sum(1)
                at += rows
    return torch.empty_like(out).index_copy_(0, order, out)


def _plane(m, include_self):
    """(neighbours, curvature, unit normal) of the covariances of _moments, by
    cyclic Jacobi rotations."""
    cnt = m[:, 0] if include_self else m[:, 0] - 1
    w = cnt.clamp(min=1)
    mu = m[:, 1:4] / w[:, None]
    a = {(i, i): m[:, 4 + i] / w - mu[:, i] ** 2 for i in range(3)}
    for k, (i, j) in enumerate(((0, 1), (0, 2), (1, 2))):
        a[i, j] = m[:, 7 + k] / w - mu[:, i] * mu[:, j]
    v = [[torch.full_like(w, float(i == j)) for j in range(3)] for i in range(3)]
    for _ in range(8):
        for i, j in ((0, 1), (0, 2), (1, 2)):
            k = 3 - i - j
            ik, jk = (min(i, k), max(i, k)), (min(j, k), max(j, k))
            off = a[i, j]
            th = (a[j, j] - a[i, i]) / torch.where(off == 0, 1.0, 2 * off)
            t = torch.where(th >= 0, 1.0, -1.0) / (th.abs() + (1 + th * th).sqrt())
            t = torch.where(off == 0, 0.0, t)
            c = 1 / (1 + t * t).sqrt()
            s = t * c
            a[i, i], a[j, j], a[i, j] = a[i, i] - t * off, a[j, j] + t * off, torch.zeros_like(off)
            a[ik], a[jk] = c * a[ik] - s * a[jk], s * a[ik] + c * a[jk]
            for row in v:
                row[i], row[j] = c * row[i] - s * row[j], s * row[i] + c * row[j]
    lam = torch.stack([a[0, 0], a[1, 1], a[2, 2]], 1)
    low = lam.argmin(1, keepdim=True)
    normal = torch.cat([torch.stack(row, 1).gather(1, low) for row in v], 1)
    total = lam.sum(1)
    curvature = torch.where(total > 0, lam.gather(1, low)[:, 0] / total, 0.0)
    return cnt, curvature, torch.nn.functional.normalize(normal, dim=1)


def _normals64(cols, radius, viewpoint, include_self=False):
    cnt, curvature, normal = _plane(_moments(cols, radius), include_self)
    to = torch.tensor(viewpoint, device=DEV, dtype=torch.float64) - torch.stack(cols, 1).double()
    if include_self:
        up = torch.tensor([0.0, 0.0, 1.0], device=DEV, dtype=torch.float64).expand_as(normal)
        normal = torch.where((cnt >= 3)[:, None], normal, up)
    normal = torch.where(((normal * to).sum(1) < 0)[:, None], -normal, normal)
    if not include_self:
        normal = torch.where((cnt >= 3)[:, None], normal, math.nan)
    return list(normal.T), torch.where(cnt >= 3, curvature, 0.0)


def _chain64(cols, leaf, radius, viewpoint):
    group, voxels, count = _voxel_groups(cols, leaf)
    means = _means(cols, group, voxels, count)
    normals, curvature = _normals64([c.float() for c in means[:3]], radius, viewpoint)
    return means + normals + [curvature]


def _padded(rows, n):
    return [torch.cat([c, c.new_zeros(n - c.shape[0])]) for c in rows]


def exact(case, seed):
    kind = case["kind"]
    n = None
    if kind in ("host", "chain", "batch", "stream"):
        cols = _inputs(case, seed)
        n = cols[0].shape[0]
    if kind == "host":
        group, voxels, count = _voxel_groups(cols, case["leaf"])
        first = _first(group, voxels)
        means = _means(cols, group, voxels, count)
        kept = 0 if case["mode"] == "approximate" else 3 if case["mode"] == "first" else len(cols)
        means[kept:] = [c[first].double() for c in cols[kept:]]
        if case["mode"] == "xyz":  # first-seen order
            order = torch.argsort(first)
            means = [c[order] for c in means]
        return dict(columns=_padded(means, n), counts=None, voxels=None)
    if kind in ("chain", "batch"):
        if kind == "batch":
            sizes, leaves = _batch_sizes(case)
            parts = [_chain64(list(c), leaf, 5.0 * leaf, VIEWPOINT)
                     for c, leaf in zip(zip(*[c.split(sizes) for c in cols]), leaves)]
            rows = [torch.cat(c) for c in zip(*parts)]
        else:
            view = (0.0, 0.0, 0.0) if case["scene"] == "lidar" else VIEWPOINT
            rows = _chain64(cols, case["leaf"], case["radius"], view)
        rows = _padded(rows, n)
        return dict(columns=rows[:-4], counts=None, normals=rows[-4:-1], curvature=rows[-1],
                    neighbors=None, voxels=None, valid=None, offsets=None)
    if kind == "normals":
        normals, curvature = _normals64(_inputs(case, seed), case["radius"], VIEWPOINT,
                                        case["include_self"])
        return dict(normals=normals, curvature=curvature, counts=None, valid=None, shell=None)
    if kind == "plane":
        cnt, _, n = _plane(_moments(_inputs(case, seed), case["radius"]), True)
        eps = 1e-3
        cov = torch.stack([1 + (eps - 1) * n[:, a] ** 2 for a in range(3)]
                          + [(eps - 1) * n[:, a] * n[:, b] for a, b in ((0, 1), (0, 2), (1, 2))], 1)
        few = torch.tensor([eps] * 3 + [0.0] * 3, device=DEV, dtype=torch.float64)
        return dict(cov=torch.where((cnt >= 3)[:, None], cov, few), valid=None)
    if kind == "las":
        f = _las_fields(case, seed)
        out = {a: f["xyz"][:, i].double() * LAS_SCALE for i, a in enumerate("xyz")}
        out.update(intensity=f["intensity"].double(), classification=None)
        _, _, gps, rgb = _las_layout(case["format"])
        if gps is not None:
            out["gps_time"] = f["gps"]
        if rgb is not None:
            out.update(red=None, green=None, blue=None)
        return out
    if kind == "stream":
        leaf = float(np.float32(case["leaf"]))
        k = [(c.double() / leaf).floor().to(torch.int64) for c in cols[:3]]
        _, group, count = torch.unique(_pack([c - c.min() for c in k]), return_inverse=True,
                                       return_counts=True)
        means = _padded(_means(cols, group, count.shape[0], count), n)
        return dict(pos=means[:3], mean=means[3:], keys=None, counts=None, voxels=None, runs=None,
                    finite=None)
    return None  # cluster: whole numbers; ransac: the winner's own float32 plane
