"""The calls this library is used for, at the sizes they come in.

Sizes and terrain follow the workloads of wolkenbase_gb300/synth.py (single
tiles of 10 thousand to 50 million points at about 100 points per square
metre, 1 mm or 1 cm quantisation, gentle to 45 degree terrain, 5 to 40%
buildings and vegetation, mixed batches); the clouds are drawn on the GPU
with the same model, because a cloud of 50 million points takes numpy tens of
seconds.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import wolkenbase_gb300 as wb
from wolkenbase_gb300 import _lib, synth

DEV = "cuda" if torch.cuda.is_available() else "cpu"
DENSITY = 100.0   # points per square metre

TERRAIN = {
    # gentle hills, 1 mm, the plain workload
    "plain": dict(scale=0.001, offset=(0.0, 0.0, 0.0), slope=None, steps=0.0, nonground=0.2),
    # slopes to 35 degrees, a third of the points on buildings and trees: the mixed batch's tiles
    "steep": dict(scale=0.001, offset=(0.0, 0.0, 0.0), slope=math.tan(math.radians(35.0)), steps=0.0, nonground=0.33),
    # UTM-like offsets at 1 cm, slopes to 45 degrees and 2 m terraces
    "utm": dict(scale=0.01, offset=(500000.0, 4500000.0, 1500.0), slope=1.0, steps=2.0, nonground=0.2),
}
LAS_BYTES = {1: 28, 3: 34, 6: 30, 7: 36}   # LAS point record lengths by format


def listed():
    return [
        # the smallest tile a request loop is asked for, numpy arrays in and class bytes out
        dict(name="request_10k", kind="classify", n=10_007, terrain="plain", pinned=False),
        # one uneven tile of a mixed batch on its own: steep, much vegetation, caller's numpy arrays
        dict(name="tile_163k_steep", kind="classify", n=163_841, terrain="steep", pinned=False),
        # the 1M-point tile of 100 x 100 m, from and to pinned host buffers
        dict(name="tile_1m", kind="classify", n=1_000_000, terrain="plain", pinned=True),
        # a LAS file's format-1 records already in HBM, with 2% of the points read twice
        dict(name="las28_5m_dups", kind="resident", n=5_000_003, terrain="steep", stride=28, dups=0.02, fp32=False),
        # the survey block of 700 x 700 m, XYZ records in HBM
        dict(name="plain_50m", kind="resident", n=50_000_000, terrain="plain", stride=12, dups=0.0, fp32=False),
        # the precision mode on steep UTM terrain
        dict(name="utm_fp32_12m", kind="resident", n=12_000_017, terrain="utm", stride=12, dups=0.0, fp32=True),
        # octree alone: leaf table and store order, for a program with queries of its own
        dict(name="build_8m", kind="build", n=8_000_009, terrain="plain", stride=12),
        # tile fit alone, on an octree that is kept while the tile size is tried out
        dict(name="scan_3m", kind="scan", n=3_000_017, terrain="utm", tile_size=1.0),
        # many uneven tiles through the server's batch call
        dict(name="batch_24", kind="batch", count=24, lo=50_000, hi=2_000_000),
        # one neighbourhood query, as a program that inspects a point asks it
        dict(name="query_2m", kind="query", n=2_000_003, shape="hyperboloid", r=0.3, sorted=True),
        # every field of a LAS file's records, as arrays in HBM
        dict(name="las_decode_8m", kind="decode", n=8_000_009, fmt=1),
        # the class-split writer: classified records into the files of their classes
        dict(name="las_write_6m", kind="write", n=6_000_011, fmt=6, per_file=1_000_000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["classify", "classify", "resident", "resident", "build", "scan", "batch", "query", "decode",
                       "write"])
    if kind == "classify":
        return dict(kind=kind, n=_log(rng, 10_000, 3_000_000), terrain=rng.choice(["plain", "steep", "utm"]),
                    pinned=rng.random() < 0.5)
    if kind == "resident":
        terrain = rng.choice(["plain", "steep", "utm"])
        return dict(kind=kind, n=_log(rng, 200_000, 40_000_000 if terrain == "plain" else 12_000_000),
                    terrain=terrain, stride=rng.choice([12, 28, 30, 34]), dups=rng.choice([0.0, 0.0, 0.02, 0.1]),
                    fp32=rng.random() < 0.25)
    if kind == "build":
        return dict(kind=kind, n=_log(rng, 50_000, 16_000_000), terrain=rng.choice(["plain", "utm"]),
                    stride=rng.choice([12, 28, 34]))
    if kind == "scan":
        return dict(kind=kind, n=_log(rng, 50_000, 6_000_000), terrain=rng.choice(["plain", "steep", "utm"]),
                    tile_size=rng.choice([0.7, 1.0, 2.0]))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(2, 32), lo=20_000, hi=_log(rng, 100_000, 2_000_000))
    if kind == "query":
        return dict(kind=kind, n=_log(rng, 20_000, 8_000_000), shape=rng.choice(["cylinder", "hyperboloid"]),
                    r=round(rng.uniform(0.1, 2.0), 3), sorted=rng.random() < 0.5)
    if kind == "decode":
        return dict(kind=kind, n=_log(rng, 10_000, 16_000_000), fmt=rng.choice(sorted(LAS_BYTES)))
    return dict(kind=kind, n=_log(rng, 50_000, 8_000_000), fmt=rng.choice(sorted(LAS_BYTES)),
                per_file=rng.choice([0, 250_000, 1_000_000]))


# ---- clouds ----

def _inside(x, y, boxes):
    hit = torch.zeros(x.shape, dtype=torch.bool, device=x.device)
    for cx, cy, hx, hy, _ in boxes:
        hit |= ((x - cx).abs() < hx) & ((y - cy).abs() < hy)
    return hit


def _terrain(n, seed, terrain, nonground=None):
    """(n, 3) int32 record integers of one square tile: four sinusoids and
    2 cm noise, box buildings with points on roofs and walls, trees in copses."""
    t = TERRAIN[terrain]
    host = np.random.default_rng(seed)
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)

    def rand(k):
        return torch.rand(k, generator=g, device=DEV, dtype=torch.float64)

    side = math.sqrt(n / DENSITY)
    amp, lam = host.uniform(0.5, 2.0, 4), host.uniform(20.0, 80.0, 4)
    th, phi = host.uniform(0.0, 2 * math.pi, 4), host.uniform(0.0, 2 * math.pi, 4)
    if t["slope"] is not None:
        amp = amp * min(1.0, t["slope"] / float(np.sum(amp * 2 * math.pi / lam)))

    def ground(x, y):
        z = torch.zeros_like(x)
        for k in range(4):
            z += amp[k] * torch.sin((x * math.cos(th[k]) + y * math.sin(th[k])) * (2 * math.pi / lam[k]) + phi[k])
        return z + t["steps"] * torch.floor((x + y) / 40.0) if t["steps"] else z

    nng = int(round((t["nonground"] if nonground is None else nonground) * n))
    nbox, nveg = nng // 2, nng - nng // 2
    ngnd = n - nng
    hmax = min(12.0, 0.15 * side)
    hmin = min(4.0, 0.5 * hmax)
    boxes = []
    for _ in range(max(1, int(round(0.1 * side * side / 256.0)))):
        hx, hy = host.uniform(hmin, hmax, 2)
        boxes.append((hx + host.random() * max(side - 2 * hx, 0.0), hy + host.random() * max(side - 2 * hy, 0.0),
                      hx, hy, host.uniform(3.0, 15.0)))

    def outside(k, place):
        xs, ys, left = [], [], k
        while left > 0:
            x, y = place(int(left * 1.3) + 64)
            keep = (x >= 0) & (x < side) & (y >= 0) & (y < side) & ~_inside(x, y, boxes)
            xs.append(x[keep][:left])
            ys.append(y[keep][:left])
            left -= xs[-1].numel()
        return torch.cat(xs), torch.cat(ys)

    gx, gy = outside(ngnd, lambda m: (rand(m) * side, rand(m) * side))
    gz = ground(gx, gy) + 0.02 * torch.randn(ngnd, generator=g, device=DEV, dtype=torch.float64)

    rmax = min(12.0, 0.2 * side)
    rmin = min(4.0, 0.5 * rmax)
    discs, area = [], 0.0
    while area < 0.15 * side * side:
        r = host.uniform(rmin, rmax)
        discs.append((host.random() * side, host.random() * side, r))
        area += math.pi * r * r
    d = torch.tensor(discs, dtype=torch.float64, device=DEV)
    cum = torch.cumsum(d[:, 2] ** 2, 0)

    def copse(m):
        k = torch.searchsorted(cum, rand(m) * cum[-1]).clamp_(max=len(discs) - 1)
        r, a = d[k, 2] * torch.sqrt(rand(m)), rand(m) * (2 * math.pi)
        return d[k, 0] + r * torch.cos(a), d[k, 1] + r * torch.sin(a)

    vx, vy = outside(nveg, copse)
    vz = ground(vx, vy) + 0.5 + 9.5 * rand(nveg)

    b = torch.tensor(boxes, dtype=torch.float64, device=DEV)
    roof_a, wall_a = 4 * b[:, 2] * b[:, 3], 4 * (b[:, 2] + b[:, 3]) * b[:, 4]
    cumb = torch.cumsum(roof_a + wall_a, 0)
    k = torch.searchsorted(cumb, rand(nbox) * cumb[-1]).clamp_(max=len(boxes) - 1)
    cx, cy, hx, hy = b[k, 0], b[k, 1], b[k, 2], b[k, 3]
    roof = ground(cx, cy) + b[k, 4]
    on_roof = rand(nbox) < (roof_a / (roof_a + wall_a))[k]
    u, v, w = 2 * rand(nbox) - 1, 2 * rand(nbox) - 1, rand(nbox)
    along_x = rand(nbox) * (hx + hy) < hx
    sign = torch.where(rand(nbox) < 0.5, -1.0, 1.0).double()
    bx = cx + torch.where(on_roof | along_x, u, sign) * hx
    by = cy + torch.where(on_roof | ~along_x, v, sign) * hy
    base = ground(bx, by)
    bz = torch.where(on_roof, roof, base + w * (roof - base).clamp(min=0.0))

    xyz = torch.stack([torch.cat([gx, bx, vx]), torch.cat([gy, by, vy]), torch.cat([gz, bz, vz])], 1)
    q = torch.round(xyz / t["scale"]).to(torch.int32)
    return q[torch.randperm(n, generator=g, device=DEV)].contiguous()


def _corners(q, t):
    """Header min/max of the records: the decoded extremes."""
    lo, hi = q.min(0).values.tolist(), q.max(0).values.tolist()
    return (tuple(t["offset"][a] + t["scale"] * lo[a] for a in range(3)),
            tuple(t["offset"][a] + t["scale"] * hi[a] for a in range(3)))


def _host_cloud(q, terrain, pinned):
    t = TERRAIN[terrain]
    mn, mx = _corners(q, t)
    if pinned:
        buf = torch.empty(q.shape, dtype=torch.int32, pin_memory=DEV == "cuda")
        buf.copy_(q)
        xyz = buf.numpy()
    else:
        xyz = q.cpu().numpy()
    return synth.Cloud(xyz, (t["scale"],) * 3, t["offset"], 1.0, mn, mx)


def _records(q, stride, seed):
    """(n, stride) LAS-like records: XYZ, then the rest of the record at random."""
    n = q.shape[0]
    if stride == 12:
        return q.view(torch.uint8).reshape(n, 12)
    g = torch.Generator(device=DEV)
    g.manual_seed(seed + 77)
    rec = torch.randint(0, 256, (n, stride), generator=g, device=DEV, dtype=torch.uint8)
    rec[:, :12] = q.view(torch.uint8).reshape(n, 12)
    return rec


def _las_records(q, fmt, seed):
    """Records of a LAS point format as a scanner writes them: 1-3 returns,
    scan angles of some 30 degrees, increasing GPS times, class 0."""
    n, length = q.shape[0], LAS_BYTES[fmt]
    rec = _records(q, length, seed)
    g = torch.Generator(device=DEV)
    g.manual_seed(seed + 78)
    nret = torch.randint(1, 4, (n,), generator=g, device=DEV)
    ret = torch.minimum(nret, torch.randint(1, 4, (n,), generator=g, device=DEV))
    if fmt < 6:
        rec[:, 14] = (ret | (nret << 3)).to(torch.uint8)
        rec[:, 15] = 0
        rec[:, 16] = torch.randint(-30, 31, (n,), generator=g, device=DEV, dtype=torch.int8).view(torch.uint8)
        gps = 20
    else:
        rec[:, 14] = (ret | (nret << 4)).to(torch.uint8)
        rec[:, 15] = 0
        rec[:, 16] = 0
        angle = torch.randint(-5000, 5001, (n, 1), generator=g, device=DEV, dtype=torch.int32).to(torch.int16)
        rec[:, 18:20] = angle.view(torch.uint8)
        gps = 22
    when = 3.0e8 + torch.arange(n, device=DEV, dtype=torch.float64) * 1e-5
    rec[:, gps:gps + 8] = when.view(torch.uint8).reshape(n, 8)
    return rec.contiguous()


def _struct(rec, n, stride, q, terrain):
    t = TERRAIN[terrain]
    mn, mx = _corners(q, t)
    return wb.cloud_struct(rec.data_ptr(), n, stride, (t["scale"],) * 3, t["offset"], 1.0, mn, mx,
                           device_resident=True)


def _check(clf, rc):
    if rc:
        raise wb.WolkenbaseError(rc, clf.L.wb_last_error(clf.ctx).decode())


def _done(**state):
    torch.cuda.synchronize()
    torch.cuda.empty_cache()   # the library allocates beside torch's cache
    return state


# ---- one pass ----

def prepare(case, seed):
    kind = case["kind"]
    if kind == "classify":
        q = _terrain(case["n"], seed, case["terrain"])
        cloud = _host_cloud(q, case["terrain"], case["pinned"])
        cls = torch.zeros(case["n"], dtype=torch.uint8, pin_memory=case["pinned"]).numpy()
        return _done(kind=kind, clf=wb.Classifier(0), cloud=cloud, params=wb.Params(), cls=cls)
    if kind == "resident":
        n = case["n"]
        q = _terrain(n, seed, case["terrain"])
        if case["dups"]:
            g = torch.Generator(device=DEV)
            g.manual_seed(seed + 5)
            k = int(case["dups"] * n)
            at = torch.randperm(n, generator=g, device=DEV)
            q[at[:k]] = q[at[k:2 * k]]
        rec = _records(q, case["stride"], seed)
        clf = wb.Classifier(0)
        if case["fp32"]:
            clf.set_precision(_lib.WB_PRECISION_FP32)
        return _done(kind=kind, clf=clf, cs=_struct(rec, n, case["stride"], q, case["terrain"]), rec=rec,
                     params=wb.Params().c(), cls=torch.zeros(n, dtype=torch.uint8, device=DEV))
    if kind == "build":
        n = case["n"]
        q = _terrain(n, seed, case["terrain"])
        rec = _records(q, case["stride"], seed)
        # the program's own arrays, with room for the most blocks it expects
        order = torch.zeros(n, dtype=torch.int32, pin_memory=True)
        room = n // 16 + 4096
        return _done(kind=kind, clf=wb.Classifier(0), cs=_struct(rec, n, case["stride"], q, case["terrain"]), rec=rec,
                     order=order, room=room, cube=np.zeros((room, 4)), first=np.zeros(room, np.int32),
                     count=np.zeros(room, np.int32))
    if kind == "scan":
        clf = wb.Classifier(0)
        clf.build(_host_cloud(_terrain(case["n"], seed, case["terrain"]), case["terrain"], False))
        return _done(kind=kind, clf=clf, params=wb.Params(tile_size=case["tile_size"]))
    if kind == "batch":
        host = np.random.default_rng(seed)
        clouds = []
        for i in range(case["count"]):
            # sizes are the case's own: the i-th of count steps over lo..hi
            f = (i + 0.5) / case["count"]
            n = int(round(math.exp(math.log(case["lo"]) * (1 - f) + math.log(case["hi"]) * f)))
            q = _terrain(n, seed + 100 * i, "steep", nonground=host.uniform(0.05, 0.40))
            clouds.append(_host_cloud(q, "steep", True))
        order = np.random.default_rng(case["count"]).permutation(case["count"])   # they arrive in no order of size
        return _done(kind=kind, srv=wb.Server(0, prep_slots=8, flush=_lib.WB_FLUSH_FULL),
                     clouds=[clouds[i] for i in order], params=wb.Params())
    if kind == "query":
        q = _terrain(case["n"], seed, "plain")
        cloud = _host_cloud(q, "plain", False)
        clf = wb.Classifier(0)
        clf.build(cloud)
        v = cloud.xyz[cloud.n // 2] * 0.001
        v = (float(v[0]), float(v[1]), float(v[2]) + 1.0)
        shape = _lib.WB_SHAPE_CYLINDER if case["shape"] == "cylinder" else _lib.WB_SHAPE_HYPERBOLOID
        return _done(kind=kind, clf=clf, shape=shape, v=v, r=case["r"], sorted=case["sorted"],
                     found=np.full(cloud.n, -1, np.int32))
    if kind == "decode":
        n, fmt = case["n"], case["fmt"]
        q = _terrain(n, seed, "utm")
        rec = _las_records(q, fmt, seed)
        as_torch = {C.c_double: torch.float64, C.c_uint16: torch.int16, C.c_uint8: torch.uint8, C.c_int32: torch.int32}
        out = {f: torch.zeros(n, dtype=as_torch[t], device=DEV) for f, t in _lib.LAS_POINT_FIELDS}
        pts = _lib.wb_las_points(**{f: t.data_ptr() for f, t in out.items()})
        return _done(kind=kind, clf=wb.Classifier(0), cs=_struct(rec, n, LAS_BYTES[fmt], q, "utm"), rec=rec, fmt=fmt,
                     out=out, pts=pts)
    n, fmt = case["n"], case["fmt"]
    q = _terrain(n, seed, "plain")
    rec = _las_records(q, fmt, seed)
    cs = _struct(rec, n, LAS_BYTES[fmt], q, "plain")
    clf = wb.Classifier(0)
    cls = torch.zeros(n, dtype=torch.uint8, device=DEV)
    _check(clf, clf.L.wb_classify_cloud(clf.ctx, C.byref(cs), C.byref(wb.Params().c()), C.c_void_p(cls.data_ptr())))
    mn, mx = _corners(q, TERRAIN["plain"])
    opt = wb.LasOutput(point_format=fmt, separate_classes=True, points_per_file=case["per_file"], min_cor=mn,
                       max_cor=mx, scale=(0.001, 0.001, 0.001), creation_day=1, creation_year=2026).c()
    out = torch.zeros((n, LAS_BYTES[fmt]), dtype=torch.uint8, device=DEV)
    return _done(kind=kind, clf=clf, cs=cs, rec=rec, cls=cls, fmt=fmt, opt=opt, out=out,
                 files=(_lib.wb_las_file * 256)(), count=C.c_int(0))


def run(s):
    kind = s["kind"]
    if kind == "classify":
        return s["clf"].classify_cloud(s["cloud"], s["params"], cls=s["cls"])
    if kind == "batch":
        return s["srv"].classify_batch(s["clouds"], s["params"])
    clf = s["clf"]
    if kind == "resident":
        _check(clf, clf.L.wb_classify_cloud(clf.ctx, C.byref(s["cs"]), C.byref(s["params"]),
                                            C.c_void_p(s["cls"].data_ptr())))
        return s["cls"]
    if kind == "build":
        clf.build_records(s["cs"])
        if clf.info()["n_leaves"] > s["room"]:
            raise MemoryError("more blocks than the program has room for")
        _check(clf, clf.L.wb_octree_leaves(clf.ctx, s["cube"].ctypes.data, s["first"].ctypes.data,
                                           s["count"].ctypes.data))
        _check(clf, clf.L.wb_octree_store_order(clf.ctx, s["order"].data_ptr()))
        return s["cube"], s["first"], s["count"], s["order"]
    if kind == "scan":
        clf.scan(s["params"])
        t = clf.tiles()
        return {f: np.ascontiguousarray(t[f]) for f in ("ex", "ey", "n_points", "tree_flags", "density", "h_scan",
                                                        "hyperboloid_size", "height")}, clf.planes()
    if kind == "query":
        got = clf.points_in(s["shape"], s["v"], s["r"], sorted=s["sorted"])
        s["found"][:got.size] = got
        return s["found"], got.size
    if kind == "decode":
        _check(clf, clf.L.wb_las_decode(clf.ctx, C.byref(s["cs"]), s["fmt"], C.byref(s["pts"])))
        return s["out"]
    _check(clf, clf.L.wb_las_write_output(clf.ctx, C.byref(s["cs"]), s["fmt"], None, C.byref(s["opt"]),
                                          C.c_void_p(s["out"].data_ptr()), 1, s["files"], 256, C.byref(s["count"])))
    points, box = np.zeros((256, 16), np.int64), np.zeros((256, 6))
    for i in range(s["count"].value):
        f = s["files"][i]
        points[i], box[i] = f.n_points, list(f.min) + list(f.max)
    return s["out"], points, box


def work(case):
    """Input read once and output written once; about 120 operations per
    classified point for its tile's sums and its nearest neighbours' tests."""
    kind = case["kind"]
    if kind in ("classify", "resident"):
        return {"bytes": 14 * case["n"], "flops": 120 * case["n"]}       # XYZ and class byte in, class byte out
    if kind == "build":
        return {"bytes": 16 * case["n"], "flops": 0}                      # XYZ in, store order out
    if kind == "scan":
        return {"bytes": 29 * case["n"], "flops": 24 * 1.2 * case["n"]}   # decoded points of 1.2 tiles each
    if kind == "batch":
        f = [(i + 0.5) / case["count"] for i in range(case["count"])]
        n = sum(int(round(math.exp(math.log(case["lo"]) * (1 - x) + math.log(case["hi"]) * x))) for x in f)
        return {"bytes": 14 * n, "flops": 120 * n}
    if kind == "query":
        # the blocks' cubes (13 bytes each, about 250 points a block) and the points found
        return {"bytes": 13 * case["n"] / 250 + 16 * DENSITY * math.pi * max(1.0, case["r"]) ** 2, "flops": 0}
    if kind == "decode":
        return {"bytes": (LAS_BYTES[case["fmt"]] + 62) * case["n"], "flops": 0}
    return {"bytes": (2 * LAS_BYTES[case["fmt"]] + 5) * case["n"], "flops": 0}


def exact(case, seed):
    """Decoded coordinates in 64 bits; classes, octree and record bytes are
    whole numbers.  Tile fits have no value of their own here: a tile at the
    cloud's edge holds one to three points, and its plane is what rounding
    leaves of a singular system."""
    if case["kind"] != "decode":
        return None
    t = TERRAIN["utm"]
    q = _terrain(case["n"], seed, "utm").cpu().numpy().astype(np.float64)
    out = {f: None for f, _ in _lib.LAS_POINT_FIELDS}
    for a, f in enumerate("xyz"):
        out[f] = torch.from_numpy(t["offset"][a] + t["scale"] * q[:, a])
    out["gps_time"] = 3.0e8 + torch.arange(case["n"], dtype=torch.float64) * 1e-5
    return out
