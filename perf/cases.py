"""What a program does with this library, case by case, over the range it is used in.

Clouds are seeded LiDAR-like tiles (rolling terrain plus 15 % canopy and building
cylinders, points in random order) made on the GPU, at the densities and sizes of the
package's own configurations: 4-40 points/m^2, 10k-10M points, leaves of 32/64/128.
Centres are cloud points picked at random, as the reference's SearchSet picks them, or
places near them.  A case is one pass through the public entry points:

  build    points on the device -> LinearOctree, its sorted cloud and its tree
  radius   neighbors / neighborsPrune of a centre set, CSR lists out
  ranges   neighborsStruct, ranges and point counts out
  hash     neighbour counts and set hashes, no lists (the every-point sweeps)
  knn      k nearest neighbours: indices, squared distances, counts
  engine   one batch of radius and kNN requests over several clouds

``api`` "device" calls the C ABI with device buffers that the program keeps, the cloud
on torch's current stream; "host" calls the Python methods with numpy arrays.
"""
import ctypes as C
import math

import numpy as np
import torch

from octrees_benchmark_b200 import LinearOctree, capi
from octrees_benchmark_b200.engine import BatchEngine, Request

CANOPY = 0.15      # share of the points in cylinders
CYLINDERS = 300
ENC = {"morton": 1, "hilbert": 5}


def _cloud(n, density, encoder="hilbert", leaf=64):
    return {"n": n, "density": density, "encoder": encoder, "leaf": leaf}


def listed():
    return [
        # a small sensor sweep that is indexed as it arrives: launches and host work count
        dict(name="build_20k", kind="build", **_cloud(20_011, 10.0, "hilbert", 32)),
        # the 1M-point Morton tile of the configurations
        dict(name="build_1M_morton", kind="build", **_cloud(1_000_000, 4.0, "morton", 128)),
        # the 10M-point Hilbert tile of the configurations
        dict(name="build_10M", kind="build", **_cloud(10_000_000, 4.444, "hilbert", 64)),
        # an interactive query: a few hundred centres from host memory, lists back to the host
        dict(name="radius_host_200", kind="radius", api="host", nq=200, shape="sphere", algo="neighborsPrune",
             r=2.5, r_hi=0.0, fp32=0, near=0.0, **_cloud(1_000_000, 4.0, "morton", 128)),
        # the 10,000-centre search set of the 1M-point configuration, larger radius
        dict(name="radius_10k", kind="radius", api="device", nq=10_000, shape="sphere", algo="neighborsPrune",
             r=5.0, r_hi=0.0, fp32=0, near=0.0, **_cloud(1_000_000, 4.0, "morton", 128)),
        # the headline radius set: 500k centres on the 10M-point tile
        dict(name="radius_500k", kind="radius", api="device", nq=500_000, shape="sphere", algo="neighborsPrune",
             r=2.5, r_hi=0.0, fp32=0, near=0.0, **_cloud(10_000_000, 4.444, "hilbert", 64)),
        # a dense scan, ground footprints of many sizes, centres beside the points
        dict(name="radius_mixed", kind="radius", api="device", nq=100_003, shape="circle", algo="neighbors",
             r=0.5, r_hi=5.0, fp32=0, near=0.5, **_cloud(2_000_000, 20.0, "hilbert", 32)),
        # ranges instead of lists, square footprint (the default kernel)
        dict(name="ranges_50k", kind="ranges", api="device", nq=50_021, shape="square", algo="neighborsStruct",
             r=5.0, r_hi=0.0, fp32=0, near=0.0, **_cloud(3_000_000, 10.0, "hilbert", 128)),
        # an interactive kNN query from host memory
        dict(name="knn_host_1k", kind="knn", api="host", nq=1_000, k=10, fp32=0, near=0.5,
             **_cloud(1_000_000, 4.0, "morton", 128)),
        # the headline kNN set: 500k centres, k = 50, on the 10M-point tile
        dict(name="knn_500k", kind="knn", api="device", nq=500_000, k=50, fp32=0, near=0.0,
             **_cloud(10_000_000, 4.444, "hilbert", 64)),
        # the long lists that feature extraction and the serving mix ask for
        dict(name="knn_k250", kind="knn", api="device", nq=30_011, k=250, fp32=0, near=0.0,
             **_cloud(5_000_000, 4.444, "hilbert", 64)),
        # a batch of the multi-cloud workload: half radius r ~ U[0.5, 5], half kNN of k 10 or 50
        dict(name="engine_16", kind="engine", clouds=16, n_lo=10_000, n_hi=2_000_000, q_lo=1_000, q_hi=200_000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["build", "build", "radius", "radius", "ranges", "hash", "knn", "knn", "knn", "engine"])
    if kind == "engine":
        return dict(kind=kind, clouds=rng.randint(2, 15), n_lo=10_000, n_hi=_log(rng, 50_000, 2_000_000), q_lo=1_000,
                    q_hi=_log(rng, 2_000, 150_000))
    cl = _cloud(_log(rng, 10_000, 10_000_000), round(rng.uniform(4.0, 40.0), 3), rng.choice(["morton", "hilbert"]),
                rng.choice([32, 64, 128]))
    if kind == "build":
        return dict(kind=kind, **cl)
    nq = _log(rng, 100, 500_000)
    api = "host" if nq < 20_000 and kind != "hash" and rng.random() < 0.4 else "device"
    near = rng.choice([0.0, 0.0, 0.5, 3.0])
    fp32 = rng.choice([0, 0, 0, 1])
    if kind == "knn":
        k = _log(rng, 1, 1000)
        return dict(kind=kind, api=api, nq=max(100, min(nq, (25_000_000 if k <= 64 else 7_000_000) // k)), k=k, fp32=fp32,
                    near=near, **cl)
    shape = rng.choice(["sphere", "sphere", "circle", "square", "cube"])
    algo = "neighborsStruct" if kind == "ranges" else rng.choice(["neighbors", "neighborsPrune"])
    r = round(rng.uniform(0.5, 10.0), 3)
    r_hi = round(r + rng.uniform(0.1, 2.5), 3) if rng.random() < 0.3 else 0.0
    c = dict(kind=kind, api=api, nq=nq, shape=shape, algo=algo, r=r, r_hi=r_hi, fp32=fp32, near=near, **cl)
    most = 2_000_000 if api == "host" else 12_000_000
    c["nq"] = int(max(50, min(nq, most / max(1.0, _mean_count(c)))))
    return c


# ---- inputs ---------------------------------------------------------------------------


def _points(n, density, seed):
    """A seeded tile: terrain of four sinusoids plus noise, and cylinders of canopy, shuffled."""
    tile = math.sqrt(n / density)
    rng = np.random.default_rng(seed)
    dirs, phases = rng.uniform(0.0, math.pi, 4), rng.uniform(0.0, 2.0 * math.pi, 4)
    g = torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)

    def rand(m):
        return torch.rand(m, dtype=torch.float64, device="cuda", generator=g)

    n_can = int(round(n * CANOPY))
    n_ter = n - n_can
    cr = np.minimum(rng.uniform(2.0, 15.0, CYLINDERS), 0.25 * tile)
    cx, cy, ch = rng.uniform(cr, tile - cr), rng.uniform(cr, tile - cr), rng.uniform(3.0, 25.0, CYLINDERS)
    cr, cx, cy, ch = (torch.from_numpy(v).cuda() for v in (cr, cx, cy, ch))
    which = torch.multinomial(cr * cr, n_can, replacement=True, generator=g)
    rad, ang = cr[which] * rand(n_can).sqrt(), rand(n_can) * (2.0 * math.pi)
    x = torch.cat([rand(n_ter) * tile, cx[which] + rad * ang.cos()])
    y = torch.cat([rand(n_ter) * tile, cy[which] + rad * ang.sin()])
    z = torch.cat([0.05 * torch.randn(n_ter, dtype=torch.float64, device="cuda", generator=g), rand(n_can) * ch[which]])
    for lam, th, ph in zip((50.0, 100.0, 200.0, 400.0), dirs, phases):
        z += 5.0 * torch.sin((2.0 * math.pi / lam) * (x * math.cos(th) + y * math.sin(th)) + ph)
    p = torch.stack([x, y, z], 1)
    return p[torch.randperm(n, device="cuda", generator=g)].contiguous(), g


def _centres(points, g, nq, near):
    sel = torch.randint(0, points.shape[0], (nq,), device="cuda", generator=g)
    c = points[sel]
    if near:
        c = c + near * (2.0 * torch.rand(c.shape, dtype=torch.float64, device="cuda", generator=g) - 1.0)
    return c.contiguous()


def _ptr(t):
    return t.data_ptr() if t is not None else None


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case, s.kind = case, case["kind"]
    if s.kind == "engine":
        return _prepare_engine(s, case, seed)
    s.points, g = _points(case["n"], case["density"], seed)
    n = case["n"]
    if s.kind == "build":
        s.keys = torch.empty(n, dtype=torch.int64, device="cuda")
        s.perm = torch.empty(n, dtype=torch.int32, device="cuda")
        s.xyz = torch.empty((n, 3), dtype=torch.float64, device="cuda")
        m = int(2.0 * _nodes(case)) + 4096  # room for the tree, kept by the program
        s.offsets = torch.zeros(m + 1, dtype=torch.int32, device="cuda")
        s.ranges = torch.zeros((m, 2), dtype=torch.int64, device="cuda")
        s.node_centers = torch.zeros((m, 3), dtype=torch.float64, device="cuda")
        return s
    nq = case["nq"]
    s.centres = _centres(s.points, g, nq, case["near"])
    s.cloud = LinearOctree(s.points, encoder=ENC[case["encoder"]], max_points_leaf=case["leaf"],
                           stream=torch.cuda.current_stream().cuda_stream, fp32_filter=case["fp32"])
    s.points = None
    if s.kind == "knn":
        k = case["k"]
        if case["api"] == "host":
            s.centres = s.centres.cpu().numpy()
        else:
            s.idx = torch.empty((nq, k), dtype=torch.int32, device="cuda")
            s.d2 = torch.empty((nq, k), dtype=torch.float64, device="cuda")
            s.cnt = torch.empty(nq, dtype=torch.int32, device="cuda")
        return s
    s.radii = None
    if case["r_hi"]:
        s.radii = case["r"] + (case["r_hi"] - case["r"]) * torch.rand(nq, dtype=torch.float64, device="cuda", generator=g)
    # the program keeps an output array with room to spare
    shape = (_room(case), 2) if s.kind == "ranges" else (_room(case),)
    if case["api"] == "host":
        s.centres = s.centres.cpu().numpy()
        s.radii = s.radii.cpu().numpy() if s.radii is not None else None
        s.out = np.zeros(shape, np.uint32)
    elif s.kind in ("radius", "ranges"):
        s.offs = torch.zeros(nq + 1, dtype=torch.int64, device="cuda")
        s.pts = torch.zeros(nq, dtype=torch.int64, device="cuda")
        s.out = torch.zeros(shape, dtype=torch.int32, device="cuda")
    return s


def _room(case):
    """Results a program makes room for: twice the expected ones, and some for the centres that are not typical."""
    return int(case["nq"] * min(case["n"], 2.0 * _mean_count(case) + 64.0)) + 65_536


def _search(s):
    """A radius or ranges call with device buffers."""
    c, h, total, cap = s.case, s.cloud.handle, C.c_uint64(0), s.out.shape[0]
    L, kern = capi.lib(), capi.KERNELS[c["shape"]]
    if s.kind == "ranges":
        st = L.oct_struct_search(h, kern, _ptr(s.centres), c["nq"], _ptr(s.radii), c["r"], _ptr(s.offs), _ptr(s.out), cap,
                                 C.byref(total), _ptr(s.pts), capi.OCT_MEM_DEVICE)
    else:
        st = L.oct_radius_search(h, kern, capi.ALGOS[c["algo"]], _ptr(s.centres), c["nq"], _ptr(s.radii), c["r"],
                                 _ptr(s.offs), _ptr(s.out), cap, C.byref(total), capi.OCT_MEM_DEVICE)
    capi.check(st, h, "search")


def _engine_sizes(case):
    """(points, centres, k) of each cloud of a batch: sizes spread evenly over their logarithm."""
    m = case["clouds"]
    for i in range(m):
        n = int(case["n_lo"] * (case["n_hi"] / case["n_lo"]) ** (i / (m - 1.0)))
        # small and large query sets fall on small and large clouds alike
        nq = int(case["q_lo"] + (case["q_hi"] - case["q_lo"]) * ((7 * i + 3) % m) / (m - 1.0))
        yield n, nq, (10, 50)[i % 2]


def _prepare_engine(s, case, seed):
    rng = np.random.default_rng(seed)
    s.engine, s.requests, s.places_at = BatchEngine(), [], []
    noff = nidx = nrow = ncnt = 0
    for i, (n, nq, k) in enumerate(_engine_sizes(case)):
        density = 4.0 + 36.0 * ((5 * i + 2) % case["clouds"]) / case["clouds"]
        pts, g = _points(n, density, int(rng.integers(0, 2**31 - 1)))
        oc = LinearOctree(pts, encoder=(1, 5)[(i // 2) % 2], max_points_leaf=(32, 64, 128)[i % 3])
        nr = nq // 2
        centres = _centres(pts, g, nq, 0.0)
        radii = 0.5 + 4.5 * torch.rand(nr, dtype=torch.float64, device="cuda", generator=g)
        s.requests += [Request(oc, "radius", centres[:nr], radii=radii, kernel="sphere", algo="neighborsPrune"),
                       Request(oc, "knn", centres[nr:], k=k)]
        room = _room(dict(n=n, density=density, nq=nr, shape="sphere", r=0.5, r_hi=5.0))
        s.places_at += [(noff, nidx, room), (nrow, ncnt)]
        noff, nidx, nrow, ncnt = noff + nr + 1, nidx + room, nrow + (nq - nr) * k, ncnt + nq - nr
    s.offs = torch.zeros(noff, dtype=torch.int64, device="cuda")
    s.idx = torch.zeros(nidx, dtype=torch.int32, device="cuda")
    s.knn_idx = torch.zeros(nrow, dtype=torch.int32, device="cuda")
    s.d2 = torch.zeros(nrow, dtype=torch.float64, device="cuda")
    s.cnt = torch.zeros(ncnt, dtype=torch.int32, device="cuda")
    return s


# ---- one pass -------------------------------------------------------------------------


def run(s):
    L, dev, c = capi.lib(), capi.OCT_MEM_DEVICE, s.case
    if s.kind == "build":
        oc = LinearOctree(s.points, encoder=ENC[c["encoder"]], max_points_leaf=c["leaf"])
        if oc.n_total >= s.offsets.shape[0]:
            raise RuntimeError("no room for the tree")
        capi.check(L.oct_encode_sort(oc.handle, None, _ptr(s.keys), _ptr(s.perm), _ptr(s.xyz), dev), oc.handle, "sorted")
        capi.check(L.oct_tree_export(oc.handle, _ptr(s.offsets), _ptr(s.ranges), _ptr(s.node_centers), None, None, dev),
                   oc.handle, "export")
        oc.close()
        return {"box": oc.box, "keys": s.keys, "perm": s.perm, "xyz": s.xyz, "offsets": s.offsets, "ranges": s.ranges,
                "centers": s.node_centers}
    if s.kind == "engine":
        places = s.engine.run(s.requests)
        e = s.engine._h
        for r, p, at in zip(s.requests, places, s.places_at):
            if r.kind == "radius":
                st = L.oct_engine_copy_radius(e, C.byref(p), _ptr(s.offs) + 8 * at[0], _ptr(s.idx) + 4 * at[1], at[2], dev)
            else:
                st = L.oct_engine_copy_knn(e, C.byref(p), r.k, _ptr(s.knn_idx) + 4 * at[0], _ptr(s.d2) + 8 * at[0],
                                           _ptr(s.cnt) + 4 * at[1], dev)
            capi.check(st, None, "copy")
        return s.offs, s.idx, s.knn_idx, s.d2, s.cnt
    if s.kind == "knn":
        if c["api"] == "host":
            return s.cloud.knn(s.centres, c["k"])
        capi.check(L.oct_knn(s.cloud.handle, _ptr(s.centres), c["nq"], c["k"], _ptr(s.idx), _ptr(s.d2), _ptr(s.cnt), dev),
                   s.cloud.handle, "knn")
        return s.idx, s.d2, s.cnt
    if s.kind == "hash":
        return s.cloud.radius_hash(s.centres, c["r"] if s.radii is None else s.radii, c["shape"], c["algo"])
    if c["api"] == "host":
        r = c["r"] if s.radii is None else s.radii
        if s.kind == "ranges":
            offs, out, pts = s.cloud.neighborsStruct(s.centres, r, c["shape"])
        else:
            offs, out = s.cloud.radius_search(s.centres, r, c["shape"], c["algo"])
        s.out[:out.shape[0]] = out
        return (offs, s.out, pts) if s.kind == "ranges" else (offs, s.out)
    _search(s)
    return (s.offs, s.out, s.pts) if s.kind == "ranges" else (s.offs, s.out)


# ---- what a pass cannot do without ----------------------------------------------------


def _mean_count(c):
    """Expected neighbours of a centre at a cloud point."""
    lo, hi = c["r"], c["r_hi"] or c["r"]
    r2 = (lo * lo + lo * hi + hi * hi) / 3.0
    area = (math.pi if c["shape"] in ("sphere", "circle") else 4.0) * r2
    tile2 = c["n"] / c["density"]
    stand = CANOPY * c["n"] / min(CYLINDERS * math.pi * 86.0, tile2)  # points per m^2 inside a cylinder
    if c["shape"] in ("sphere", "cube"):  # they reach over part of a cylinder's height
        stand *= min(1.0, (1.2 if c["shape"] == "sphere" else 2.0) * math.sqrt(r2) / 14.0)
    return min(c["n"], area * (c["density"] + CANOPY * stand))


def _search_bytes(n, nq, reached, out_bytes):
    return 24.0 * nq + 24.0 * min(n, nq * reached) + out_bytes


def _nodes(case):
    """Expected nodes of a tree."""
    return 8.0 / 7.0 * case["n"] / (0.22 * case["leaf"])


def work(case):
    kind = case["kind"]
    if kind == "build":
        n, nodes = case["n"], _nodes(case)
        # points in; keys, ids and points out; a tree of 36 bytes a node (44 as exported)
        return {"bytes": 24.0 * n + (8.0 + 4.0 + 24.0) * n + 44.0 * nodes, "flops": 30.0 * n}
    if kind == "engine":
        total = {"bytes": 0.0, "flops": 0.0}
        for i, (n, nq, k) in enumerate(_engine_sizes(case)):
            m = _mean_count(dict(n=n, density=4.0 + 36.0 * ((5 * i + 2) % case["clouds"]) / case["clouds"], shape="sphere",
                                 r=0.5, r_hi=5.0))
            total["bytes"] += _search_bytes(n, nq, 0.5 * (m + k), 0.5 * nq * (8.0 + 4.0 * m + 12.0 * k + 4.0))
            total["flops"] += 4.0 * nq * (m + k)
        return total
    n, nq = case["n"], case["nq"]
    if kind == "knn":
        k = min(case["k"], n)
        return {"bytes": _search_bytes(n, nq, k, nq * (12.0 * k + 4.0)), "flops": 8.0 * nq * k}
    m = _mean_count(case)
    if kind == "hash":
        out = 16.0 * nq
    elif kind == "ranges":
        out = nq * (16.0 + 8.0 * m / 12.0)
    else:
        out = nq * (8.0 + 4.0 * m)
    return {"bytes": _search_bytes(n, nq, m, out), "flops": 8.0 * nq * m}


# ---- the same in 64 bits, without this package's search ------------------------------


def exact(case, seed):
    if case["kind"] == "build":
        p, _ = _points(case["n"], case["density"], seed)
        lo, hi = p.amin(0).cpu().numpy(), p.amax(0).cpu().numpy()
        mid, rad = 0.5 * (lo + hi), 0.5 * (hi - lo)
        return {"box": np.concatenate([mid, rad, mid - rad, mid + rad]), "keys": None, "perm": None, "xyz": None,
                "offsets": None, "ranges": None, "centers": None}
    if case["kind"] != "knn" or float(case["n"]) * case["nq"] > 3e10:
        return None
    p, g = _points(case["n"], case["density"], seed)
    q = _centres(p, g, case["nq"], case["near"])
    k, m = case["k"], min(case["k"], case["n"])
    d2 = torch.full((case["nq"], k), math.inf, dtype=torch.float64, device="cuda")
    step = max(1, 100_000_000 // case["n"])
    for a in range(0, case["nq"], step):
        b = q[a:a + step]
        d = (b[:, :1] - p[:, 0]) ** 2
        d += (b[:, 1:2] - p[:, 1]) ** 2
        d += (b[:, 2:] - p[:, 2]) ** 2
        d2[a:a + step, :m] = torch.topk(d, m, dim=1, largest=False, sorted=True).values
    return (None, d2, None) if case["api"] == "device" else (None, d2.cpu().numpy(), None)
