"""The calls that users of this library make, at the sizes they make them: the
workloads its performance is measured on.

A case is a dict of plain values.  ``listed()`` names the standing ones,
``draw(rng)`` gives further ones of the same ranges, ``prepare(case, seed)``
makes what a program has in hand before the call (a built tree, its inputs and
output buffers), ``run(state)`` is one pass through the public entry points of
``ikd-tree_gb300/ikdg.py`` and ``work(case)`` counts what such a pass cannot do
without.  ``exact(case, seed)`` gives computed outputs in 64 bits.

Kinds:

  knn       Nearest_Search of a batch of queries; ``io`` says where its buffers
            are: "device" (asynchronous), "pinned" (page-locked host buffers
            kept by the caller) or "host" (ordinary arrays)
  box       Box_Search of a batch of boxes, ids and points out
  radius    Radius_Search of a batch of centres, ids and points out
  batch     one run of a batch of kNN, box and radius requests on many trees
  build     Build of a map, then the first scan's search on it
  update    one LiDAR scan of a mapping loop: Nearest_Search of the scan,
            Add_Points with voxel downsampling, Delete_Point_Boxes of all that
            left the sliding cube
  edit      a local map edit: Delete_Point_Boxes of some boxes, Add_Points of
            their points and of new ones, a search, Delete_Points of the new
            ones (the stored set is the same after every pass)
  register  the scan-to-map step: point-to-plane residuals and their adjoint

Maps: "uniform" points in [-50, 50]^3 m; "lidar", a ground plane of 400 x 400 m
and 200 walls with 2 cm noise; "slab", points in [-500, 500]^2 x [0, 50] m of
which a third lies on planar patches.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ikd-tree_gb300"))

import ikdg  # noqa: E402

EXTENT = 50.0        # uniform maps span [-EXTENT, EXTENT]^3
GROUND = 200.0       # the LiDAR world's ground spans [-GROUND, GROUND]^2
WALLS = 200
BEAMS = 32
SENSOR_H = 1.8
CUBE = 100.0         # half side of the sliding cube that a mapping loop keeps
RETURNS = 23         # points per scan column that the mapping loop gets
SCANS = 48           # scans of a prepared drive; the loop goes along it and back
SIDE = (0.5, 5.0)    # box sides and radii of the range searches, m


def listed():
    return [
        # a front end that searches point by point: the smallest call there is
        dict(name="knn_point_host", kind="knn", map="uniform", n=1_000_000, nq=1, k=5, max_dist=-1.0, io="host"),
        # one LiDAR scan against a 2M-point map, the search of every odometry iteration
        dict(name="knn_scan_host", kind="knn", map="lidar", n=2_000_000, nq=15_000, k=5, max_dist=5.0, io="host"),
        # the standard batch: 100k queries, k = 5, buffers on the GPU ...
        dict(name="knn_batch_device", kind="knn", map="uniform", n=1_000_000, nq=100_000, k=5, max_dist=-1.0,
             io="device"),
        # ... and end to end from page-locked host buffers
        dict(name="knn_batch_pinned", kind="knn", map="uniform", n=1_000_000, nq=100_000, k=5, max_dist=-1.0,
             io="pinned"),
        # a city-sized map and a large k (normal estimation, outlier filters)
        dict(name="knn_large_k16", kind="knn", map="slab", n=20_000_000, nq=1_000_000, k=16, max_dist=2.0,
             io="device"),
        # crops: many small boxes around points of interest
        dict(name="box_batch", kind="box", n=1_000_000, nq=100_000, io="device"),
        # neighbourhoods of a fixed radius (features, clustering); radii differ by ten, hits by a thousand
        dict(name="radius_batch", kind="radius", n=1_000_000, nq=100_000, io="device"),
        # many independent maps (fleet, submaps), all their requests at once
        dict(name="batch_maps", kind="batch", maps=64, n_lo=10_000, n_hi=1_000_000, q_lo=1_000, q_hi=100_000),
        # loading a map
        dict(name="build_map", kind="build", map="lidar", n=2_000_000),
        # the mapping loop at 20k rays per scan
        dict(name="update_scan", kind="update", n=2_000_000, azimuths=625, voxel=0.5),
        # small edits of a small map: launches and host work count
        dict(name="edit_small", kind="edit", n=100_000, m=1_000, boxes=10, side_lo=2.0, side_hi=10.0, nq=1_000),
        # the differentiable registration step, forward and backward
        dict(name="register_scan", kind="register", n=1_000_000, nq=20_000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["knn", "knn", "knn", "box", "radius", "batch", "build", "update", "edit", "register"])
    if kind == "knn":
        c = dict(kind=kind, map=rng.choice(["uniform", "uniform", "lidar"]), n=_log_int(rng, 10_000, 3_000_000),
                 nq=_log_int(rng, 1, 300_000), k=rng.choice([1, 2, 3, 5, 5, 8, 10, 16, 20, 32]),
                 max_dist=rng.choice([-1.0, 1.0, 5.0]), io=rng.choice(["device", "device", "host", "pinned"]))
        if c["map"] == "lidar":
            c["nq"] = min(c["nq"], 15_000)  # a scan
        return c
    if kind in ("box", "radius"):
        io = rng.choice(["device", "device", "device", "host"])
        return dict(kind=kind, n=_log_int(rng, 10_000, 1_000_000), io=io,
                    nq=_log_int(rng, 1, 2_000 if io == "host" else 100_000))
    if kind == "batch":
        return dict(kind=kind, maps=rng.randint(3, 48), n_lo=10_000, n_hi=_log_int(rng, 50_000, 1_000_000), q_lo=1_000,
                    q_hi=_log_int(rng, 5_000, 100_000))
    if kind == "build":
        return dict(kind=kind, map=rng.choice(["uniform", "lidar"]), n=_log_int(rng, 5_000, 2_000_000))
    if kind == "update":
        return dict(kind=kind, n=_log_int(rng, 200_000, 2_000_000), azimuths=rng.randint(101, 625),
                    voxel=round(rng.uniform(0.2, 1.0), 2))
    if kind == "edit":
        return dict(kind=kind, n=_log_int(rng, 20_000, 1_000_000), m=_log_int(rng, 50, 5_000), boxes=rng.randint(1, 40),
                    side_lo=2.0, side_hi=10.0, nq=_log_int(rng, 100, 4_000))
    return dict(kind=kind, n=_log_int(rng, 100_000, 1_000_000), nq=_log_int(rng, 2_000, 20_000))


# ---- inputs --------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _u(g, shape, lo, hi):
    """Uniform float64 values on the GPU."""
    return torch.rand(shape, generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo


def _normal(g, shape, sigma):
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.float64) * sigma


def _host(t):
    return t.to(torch.float32).cpu().numpy()


def _uniform(g, n):
    return _u(g, (n, 3), -EXTENT, EXTENT)


def _world(g):
    return dict(c=_u(g, (WALLS, 2), -GROUND, GROUND), yaw=_u(g, (WALLS,), 0, math.pi), len=_u(g, (WALLS,), 2, 30),
                h=_u(g, (WALLS,), 3, 15))


def _lidar_map(w, g, n):
    """n samples of the ground and the walls in proportion to their areas."""
    area = torch.cat([torch.full((1,), (2 * GROUND) ** 2, device="cuda", dtype=torch.float64), w["len"] * w["h"]])
    which = torch.multinomial(area, n, replacement=True, generator=g) - 1
    wall = which.clamp(min=0)
    s = _u(g, (n,), -0.5, 0.5) * w["len"][wall]
    h = _u(g, (n,), 0, 1) * w["h"][wall]
    on_wall = torch.stack([w["c"][wall, 0] + s * torch.cos(w["yaw"][wall]),
                           w["c"][wall, 1] + s * torch.sin(w["yaw"][wall]), h], 1)
    ground = torch.cat([_u(g, (n, 2), -GROUND, GROUND), torch.zeros((n, 1), device="cuda", dtype=torch.float64)], 1)
    return torch.where((which < 0)[:, None], ground, on_wall) + _normal(g, (n, 3), 0.02)


def _scan(w, g, x, y, yaw, azimuths):
    """The returns of one turn of a 32-beam scanner (elevation -15..+15
    degrees, range 1-100 m, 2 cm noise) at (x, y), in the world frame."""
    f8 = dict(device="cuda", dtype=torch.float64)
    el = torch.linspace(-15, 15, BEAMS, **f8).deg2rad()[:, None]
    az = (yaw + 2 * math.pi * torch.arange(azimuths, **f8) / azimuths)[None, :]
    d = torch.stack([torch.cos(el) * torch.cos(az), torch.cos(el) * torch.sin(az), torch.sin(el).expand(-1, azimuths)],
                    -1).reshape(-1, 3)
    o = torch.tensor([x, y, SENSOR_H], **f8)
    inf = torch.tensor(math.inf, **f8)
    t = torch.where(d[:, 2] < 0, -o[2] / d[:, 2], inf)
    hit = o + torch.where(torch.isfinite(t), t, torch.zeros_like(t))[:, None] * d
    t = torch.where((hit[:, 0].abs() > GROUND) | (hit[:, 1].abs() > GROUND), inf, t)
    nx, ny, ux, uy = -torch.sin(w["yaw"]), torch.cos(w["yaw"]), torch.cos(w["yaw"]), torch.sin(w["yaw"])
    tw = ((w["c"][:, 0] - x) * nx + (w["c"][:, 1] - y) * ny)[None] / (d[:, :1] * nx + d[:, 1:2] * ny)
    along = (x + tw * d[:, :1] - w["c"][:, 0]) * ux + (y + tw * d[:, 1:2] - w["c"][:, 1]) * uy
    z = SENSOR_H + tw * d[:, 2:3]
    ok = (tw > 0) & (along.abs() <= w["len"] / 2) & (z >= 0) & (z <= w["h"])
    t = torch.minimum(t, torch.where(ok, tw, inf).amin(1))
    keep = (t >= 1.0) & (t <= 100.0)
    r = t[keep] + _normal(g, (int(keep.sum()),), 0.02)
    return o + r[:, None] * d[keep]


def _slab(g, n):
    nc = n // 3
    p = _u(g, (n, 3), 0, 1) * torch.tensor([1000.0, 1000.0, 50.0], device="cuda") - torch.tensor(
        [500.0, 500.0, 0.0], device="cuda")
    which = torch.randint(0, 400, (nc,), generator=g, device="cuda")
    centre = _u(g, (400, 3), 0, 1) * torch.tensor([1000.0, 1000.0, 50.0], device="cuda") - torch.tensor(
        [500.0, 500.0, 0.0], device="cuda")
    a = torch.nn.functional.normalize(_normal(g, (400, 3), 1.0), dim=1)
    b = torch.nn.functional.normalize(torch.linalg.cross(a, _normal(g, (400, 3), 1.0)), dim=1)
    size = _u(g, (400, 2), 10, 60)
    s = _u(g, (nc, 2), -0.5, 0.5) * size[which]
    p[:nc] = centre[which] + s[:, :1] * a[which] + s[:, 1:] * b[which] + _normal(g, (nc, 3), 0.02)
    return p[torch.randperm(n, generator=g, device="cuda")]


def _map_and_queries(case, g):
    """Map points and kNN queries, float32 on the GPU."""
    if case["map"] == "uniform":
        p, q = _uniform(g, case["n"]), _uniform(g, case["nq"])
    elif case["map"] == "slab":
        p = _slab(g, case["n"])
        q = _u(g, (case["nq"], 3), 0, 1) * torch.tensor([1000.0, 1000.0, 50.0], device="cuda") - torch.tensor(
            [500.0, 500.0, 0.0], device="cuda")
    else:
        w = _world(g)
        p = _lidar_map(w, g, case["n"])
        q = _scan(w, g, 0.0, 0.0, 0.3, 625)
        while len(q) < case["nq"]:  # a scene with few returns: the next turn's too
            q = torch.cat([q, _scan(w, g, 1.0, 0.0, 0.4, 625)])
        # the first nq returns of an evenly thinned scan, in scan order
        q = q[(torch.arange(case["nq"], device="cuda") * len(q)) // max(case["nq"], 1)]
    return p.float(), q.float().contiguous()


def _max_dist(case):
    return math.inf if case["max_dist"] < 0 else case["max_dist"]


def _tree(points, voxel=0.5):
    t = ikdg.KDTree(0.5, 0.6, voxel)
    t.Build(_host(points))
    return t


def _dev(shape, dtype):
    return torch.zeros(shape, dtype=dtype, device="cuda")


def _range_inputs(case, g):
    c = _uniform(g, case["nq"])
    if case["kind"] == "box":
        s = _u(g, (case["nq"], 3), *SIDE) / 2
        return torch.cat([c - s, c + s], 1).float(), None
    return c.float(), _u(g, (case["nq"],), *SIDE).float()


# ---- prepare ---------------------------------------------------------------------


def prepare(case, seed):
    g = _gen(seed)
    st = globals()["_prepare_" + case["kind"]](case, g)
    st["case"] = case
    torch.cuda.synchronize()
    return st


def _prepare_knn(case, g):
    p, q = _map_and_queries(case, g)
    nq, k = case["nq"], case["k"]
    st = dict(tree=_tree(p))
    if case["io"] == "host":
        st["q"] = q.cpu().numpy()
        return st
    if case["io"] == "pinned":
        def buf(shape, dtype):
            return torch.zeros(shape, dtype=dtype).pin_memory()
        st["q"] = q.cpu().pin_memory()
    else:
        buf = _dev
        st["q"] = q
    st.update(ids=buf((nq, k), torch.int32), d2=buf((nq, k), torch.float32), xyz=buf((nq, k, 3), torch.float32),
              cnt=buf((nq,), torch.int32))
    return st


def _prepare_box(case, g):
    tree = _tree(_uniform(g, case["n"]))
    q, r = _range_inputs(case, g)
    if case["io"] == "host":
        return dict(tree=tree, q=q.cpu().numpy(), r=None if r is None else r.cpu().numpy())
    cap = _capacity(case["n"], (2 * EXTENT) ** 3, case["nq"], 3 if case["kind"] == "box" else 0)
    return dict(tree=tree, q=q, r=r, cap=cap, offs=_dev((case["nq"] + 1,), torch.int64), total=_dev((1,), torch.int64),
                ids=_dev((cap,), torch.int32), xyz=_dev((cap, 3), torch.float32))


_prepare_radius = _prepare_box


def _capacity(n, volume, nq, box):
    """Room for the results of nq range queries: what they are expected to hold
    and eight standard deviations of it (most of the spread is the sizes')."""
    most = min(n, n * SIDE[1] ** 3 * (1.0 if box else 4 * math.pi / 3) / volume)
    return int(1.05 * _hits(n, volume, nq, box) + 4 * math.sqrt(nq) * most + 4096)


def _range_call(case, st):
    ids, xyz = st["ids"].data_ptr(), st["xyz"].data_ptr()
    if case["kind"] == "box":
        st["tree"].box_search_device(st["q"].data_ptr(), case["nq"], st["offs"].data_ptr(), ids, st["cap"], xyz,
                                     st["total"].data_ptr())
    else:
        st["tree"].radius_search_device(st["q"].data_ptr(), case["nq"], st["r"].data_ptr(), st["offs"].data_ptr(), ids,
                                        st["cap"], xyz, st["total"].data_ptr())


def _batch_sizes(case):
    """Per map: points, queries of each kind, k, max_dist and sides.  Sizes are
    spread evenly over the logarithm; larger maps do not get the larger query
    batches; sides are spread evenly over 20-200 m (low-discrepancy steps)."""
    m = case["maps"]
    out = []
    for i in range(m):
        f = i / max(m - 1, 1)
        j = (i * 37 + 11) % m / max(m - 1, 1)
        n = int(round(case["n_lo"] * (case["n_hi"] / case["n_lo"]) ** f))
        nq = int(round(case["q_lo"] * (case["q_hi"] / case["q_lo"]) ** j))
        nk, nb = int(round(0.6 * nq)), int(round(0.2 * nq))
        side = [20.0 + 180.0 * (((i + 1) * s) % 1.0) for s in (0.6180339887, 0.7548776662, 0.5698402910)]
        out.append(dict(n=n, nk=nk, nb=nb, nr=nq - nk - nb, k=1 + (i * 7) % 16, max_dist=1.0 + 9.0 * (i % 10) / 9.0,
                        side=side))
    return out


def _prepare_batch(case, g):
    sizes = _batch_sizes(case)
    b = ikdg.Batch()
    ins, rng_req, trees = [], [], []
    nk = sum(s["nk"] * s["k"] for s in sizes)
    out = dict(ids=_dev((nk,), torch.int32), d2=_dev((nk,), torch.float32), xyz=_dev((nk, 3), torch.float32),
               cnt=_dev((sum(s["nk"] for s in sizes),), torch.int32))
    at = at_q = 0
    for s in sizes:
        lo = _u(g, (3,), -500.0, 500.0)
        side = torch.tensor(s["side"], device="cuda", dtype=torch.float64)
        t = _tree(lo + _u(g, (s["n"], 3), 0, 1) * side)
        trees.append(t)
        q = (lo + _u(g, (s["nk"], 3), 0, 1) * side).float()
        c = lo + _u(g, (s["nb"], 3), 0, 1) * side
        half = _u(g, (s["nb"], 1), *SIDE) / 2
        box = torch.cat([c - half, c + half], 1).float()
        cen = (lo + _u(g, (s["nr"], 3), 0, 1) * side).float()
        rad = _u(g, (s["nr"],), *SIDE).float()
        ins += [q, box, cen, rad]
        b.add_knn(t, q.data_ptr(), s["nk"], s["k"], s["max_dist"], out["ids"][at:].data_ptr(), out["d2"][at:].data_ptr(),
                  out["xyz"][at:].data_ptr(), out["cnt"][at_q:].data_ptr())
        at += s["nk"] * s["k"]
        at_q += s["nk"]
        vol = s["side"][0] * s["side"][1] * s["side"][2]
        rng_req.append(("box", t, box, None, s["nb"], _capacity(s["n"], vol, s["nb"], 1)))
        rng_req.append(("radius", t, cen, rad, s["nr"], _capacity(s["n"], vol, s["nr"], 0)))
    room = sum(r[5] for r in rng_req)
    out.update(offs=_dev((sum(r[4] + 1 for r in rng_req),), torch.int64), range_ids=_dev((room,), torch.int32),
               range_xyz=_dev((room, 3), torch.float32))
    at = at_o = 0
    for kind, t, q, r, m, cap in rng_req:
        o, i, x = out["offs"][at_o:].data_ptr(), out["range_ids"][at:].data_ptr(), out["range_xyz"][at:].data_ptr()
        if kind == "box":
            b.add_box_search(t, q.data_ptr(), m, o, i, cap, x)
        else:
            b.add_radius_search(t, q.data_ptr(), m, r.data_ptr(), o, i, cap, x)
        at += cap
        at_o += m + 1
    return dict(batch=b, trees=trees, ins=ins, out=out, n_range=len(rng_req))


def _prepare_build(case, g):
    p, q = _map_and_queries(dict(case, nq=8000), g)
    return dict(tree=ikdg.KDTree(0.5, 0.6, 0.5), p=p.cpu().numpy(), q=q.cpu().numpy())


def _cube(x, y):
    """Everything outside the cube around (x, y), as six boxes."""
    far = 1.0e9
    lo, hi = (x - CUBE, y - CUBE, SENSOR_H - CUBE), (x + CUBE, y + CUBE, SENSOR_H + CUBE)
    return np.asarray([[-far, -far, -far, lo[0], far, far], [hi[0], -far, -far, far, far, far],
                       [lo[0], -far, -far, hi[0], lo[1], far], [lo[0], hi[1], -far, hi[0], far, far],
                       [lo[0], lo[1], -far, hi[0], hi[1], lo[2]], [lo[0], lo[1], hi[2], hi[0], hi[1], far]], np.float32)


def _prepare_update(case, g):
    w = _world(g)
    tree = _tree(_lidar_map(w, g, case["n"]), case["voxel"])
    turns = _normal(g, (SCANS,), 0.1).cpu().tolist()
    x = y = yaw = 0.0
    scans = []
    for s in range(SCANS):
        q = _scan(w, g, x, y, yaw, case["azimuths"])
        # thinned to a fixed size: about 24 rays of a column return
        q = q[(torch.arange(RETURNS * case["azimuths"], device="cuda") * len(q)) // (RETURNS * case["azimuths"])]
        scans.append((_host(q), _cube(x, y)))
        yaw += turns[s]
        x, y = x + math.cos(yaw), y + math.sin(yaw)
    tree.Delete_Point_Boxes(scans[0][1])  # the loop is under way: the map is the cube's already
    return dict(tree=tree, scans=scans + scans[-2:0:-1], at=0)


def _prepare_edit(case, g):
    p = _uniform(g, case["n"]).float()
    tree = _tree(p)
    sets = []
    for _ in range(16):
        c = _uniform(g, case["boxes"])
        s = _u(g, (case["boxes"], 3), case["side_lo"], case["side_hi"]) / 2
        box = torch.cat([c - s, c + s], 1).float()
        hit = ((p[:, None, :] >= box[None, :, :3]) & (p[:, None, :] < box[None, :, 3:])).all(2).any(1)
        new = _uniform(g, case["m"]).float()
        # boxes; their points and the new ones to insert; the new ones again, to delete; queries
        sets.append((box.cpu().numpy(), torch.cat([p[hit], new]).cpu().numpy(), new.cpu().numpy(),
                     _host(_uniform(g, case["nq"]))))
    return dict(tree=tree, sets=sets, at=0)


def _pose(g):
    """A pose perturbed by 2 degrees and 0.3 m."""
    return (_normal(g, (3,), math.radians(2.0)).cpu().tolist() + _normal(g, (3,), 0.3).cpu().tolist())


def _register_inputs(case, g):
    w = _world(g)
    p = _lidar_map(w, g, case["n"]).float()
    q = _scan(w, g, 0.0, 0.0, 0.3, 1000)
    while len(q) < case["nq"]:
        q = torch.cat([q, _scan(w, g, 1.0, 0.0, 0.4, 1000)])
    q = q[(torch.arange(case["nq"], device="cuda") * len(q)) // case["nq"]].float().contiguous()
    return p, q, _pose(g)


def _prepare_register(case, g):
    p, q, pose = _register_inputs(case, g)
    n = case["nq"]
    return dict(tree=_tree(p), q=q, pose=pose, planes=_dev((n, 8), torch.float32), res=_dev((n,), torch.float32),
                valid=_dev((n,), torch.int32), grad=_dev((n, 3), torch.float32))


# ---- run ----------------------------------------------------------------------------


def run(state):
    return globals()["_run_" + state["case"]["kind"]](state["case"], state)


def _run_knn(case, st):
    t, k, md = st["tree"], case["k"], _max_dist(case)
    if case["io"] == "host":
        ids, d2, xyz, cnt = t.knn(st["q"], k, md)
        return dict(ids=ids, d2=d2, xyz=xyz, cnt=cnt)
    call = t.knn_into if case["io"] == "pinned" else t.knn_device
    call(st["q"].data_ptr(), case["nq"], k, md, st["ids"].data_ptr(), st["d2"].data_ptr(), st["xyz"].data_ptr(),
         st["cnt"].data_ptr())
    return dict(ids=st["ids"], d2=st["d2"], xyz=st["xyz"], cnt=st["cnt"])


def _run_box(case, st):
    if case["io"] == "host":
        offs, ids, xyz = (st["tree"].box_search(st["q"]) if case["kind"] == "box"
                          else st["tree"].radius_search(st["q"], st["r"]))
        return dict(offs=offs, ids=ids, xyz=xyz)
    _range_call(case, st)
    return dict(offs=st["offs"], total=st["total"], ids=st["ids"], xyz=st["xyz"])


_run_radius = _run_box


def _run_batch(case, st):
    st["batch"].run()
    totals = st["batch"].synchronize(st["n_range"])  # tells whether every request's results fitted
    return dict(st["out"], totals=totals)


def _run_build(case, st):
    st["tree"].Build(st["p"])
    ids, d2, xyz, cnt = st["tree"].knn(st["q"], 5, 5.0)
    return dict(ids=ids, d2=d2, xyz=xyz, cnt=cnt, box=st["tree"].tree_range(), size=st["tree"].size())


def _run_update(case, st):
    pts, boxes = st["scans"][st["at"]]
    st["at"] = (st["at"] + 1) % len(st["scans"])
    ids, d2, xyz, cnt = st["tree"].knn(pts, 5, 5.0)
    added = st["tree"].Add_Points(pts, True)
    deleted = st["tree"].Delete_Point_Boxes(boxes)
    return dict(ids=ids, d2=d2, xyz=xyz, cnt=cnt, added=added, deleted=deleted, valid=st["tree"].validnum())


def _run_edit(case, st):
    boxes, back, new, q = st["sets"][st["at"]]
    st["at"] = (st["at"] + 1) % len(st["sets"])
    t = st["tree"]
    deleted = t.Delete_Point_Boxes(boxes)
    t.Add_Points(back, False)
    ids, d2, xyz, cnt = t.knn(q, 5)
    t.Delete_Points(new)
    return dict(ids=ids, d2=d2, xyz=xyz, cnt=cnt, deleted=deleted, valid=t.validnum())


def _run_register(case, st):
    t, n = st["tree"], case["nq"]
    ptrs = (st["planes"].data_ptr(), st["res"].data_ptr(), st["valid"].data_ptr())
    loss = t.p2p_forward(st["q"].data_ptr(), n, st["pose"], 5, 5.0, 0.1, *ptrs)
    grad_pose = t.p2p_adjoint(st["q"].data_ptr(), n, st["pose"], *ptrs, 1.0, st["grad"].data_ptr())
    return dict(loss=loss, grad_pose=np.asarray(grad_pose), planes=st["planes"], res=st["res"], valid=st["valid"],
                grad=st["grad"])


# ---- work ------------------------------------------------------------------------------


def _knn_work(n, nq, k):
    """Queries in, rows out, and each neighbour's point read (no more than the
    whole map)."""
    return 12 * nq + 20 * k * nq + 4 * nq + min(16 * n, 16 * k * nq), 8 * k * nq


def _hits(n, volume, nq, box):
    """Expected hits of nq range queries on n points in `volume`; box: 3, boxes
    of three independent sides; 1, cubes; 0, balls."""
    lo, hi = SIDE
    mean = (((lo + hi) / 2) ** 3 if box == 3 else
            (hi**4 - lo**4) / (4 * (hi - lo)) * (1.0 if box else 4 * math.pi / 3))
    return nq * min(n, n * mean / volume)


def _range_work(n, volume, nq, box):
    """Queries in, offsets and the expected hits out, each hit's point read."""
    hits = _hits(n, volume, nq, box)
    return (24 if box else 16) * nq + 8 * nq + 16 * hits + min(16 * n, 16 * hits), 8 * hits


def work(case):
    kind = case["kind"]
    if kind == "knn":
        b, f = _knn_work(case["n"], case["nq"], case["k"])
    elif kind in ("box", "radius"):
        b, f = _range_work(case["n"], (2 * EXTENT) ** 3, case["nq"], 3 if kind == "box" else 0)
    elif kind == "batch":
        b = f = 0
        for s in _batch_sizes(case):
            vol = s["side"][0] * s["side"][1] * s["side"][2]
            for x, y in (_knn_work(s["n"], s["nk"], s["k"]), _range_work(s["n"], vol, s["nb"], 1),
                         _range_work(s["n"], vol, s["nr"], 0)):
                b, f = b + x, f + y
    elif kind == "build":
        # points in, stored points and one 64-byte record per 16 points out
        b, f = (12 + 16 + 4) * case["n"], 3 * case["n"]
    elif kind == "update":
        m = RETURNS * case["azimuths"]
        b, f = _knn_work(case["n"], m, 5)
        b, f = b + 12 * m + 32 * m + 6 * 24, f + 20 * m
    elif kind == "edit":
        b, f = _knn_work(case["n"], case["nq"], 5)
        hit = case["n"] * case["boxes"] * ((case["side_lo"] + case["side_hi"]) / 2) ** 3 / (2 * EXTENT) ** 3
        b += 24 * case["boxes"] + 28 * (hit + case["m"]) + 16 * hit + 28 * case["m"]
    else:
        n = case["nq"]
        b, f = 12 * n + min(16 * case["n"], 80 * n) + 52 * n + 44 * n, 400 * n
    return {"bytes": b, "flops": f}


# ---- exact -----------------------------------------------------------------------------

MOST_PAIRS = 4.1e10  # brute force over more (query, point) pairs takes too long


def _nearest(p, q, k, max_sq):
    """Distances (ascending) and indices of the k nearest of p, in 64 bits."""
    p, q = p.double(), q.double()
    k = min(k, len(p))
    step = max(1, int(1.5e8) // len(p))
    ds, js = [], []
    for i in range(0, len(q), step):
        d = (q[i:i + step, None, 0] - p[None, :, 0]) ** 2
        for a in (1, 2):
            d += (q[i:i + step, None, a] - p[None, :, a]) ** 2
        v, j = torch.topk(d, k, dim=1, largest=False)
        ds.append(v)
        js.append(j)
    d, j = torch.cat(ds), torch.cat(js)
    return torch.where(d <= max_sq, d, torch.full_like(d, math.inf)), j


def exact(case, seed):
    g = _gen(seed)
    if case["kind"] == "knn":
        if float(case["n"]) * case["nq"] > MOST_PAIRS:
            return None
        p, q = _map_and_queries(case, g)
        d, _ = _nearest(p, q, case["k"], _max_dist(case) ** 2)
        full = torch.full((case["nq"], case["k"]), math.inf, dtype=torch.float64, device="cuda")
        full[:, :d.shape[1]] = d
        return dict(ids=None, d2=full, xyz=None, cnt=None)
    if case["kind"] == "register":
        return _exact_register(case, g)
    return None


def _exact_register(case, g):
    p, q, pose = _register_inputs(case, g)
    f8 = dict(device="cuda", dtype=torch.float64)
    om, t = torch.tensor(pose[:3], **f8), torch.tensor(pose[3:], **f8)
    th = float(om.norm())
    K = torch.tensor([[0, -pose[2], pose[1]], [pose[2], 0, -pose[0]], [-pose[1], pose[0], 0]], **f8)
    eye = torch.eye(3, **f8)
    R = eye + math.sin(th) / th * K + (1 - math.cos(th)) / th**2 * (K @ K)
    J = eye - (1 - math.cos(th)) / th**2 * K + (th - math.sin(th)) / th**3 * (K @ K)
    w = q.double() @ R.T + t
    d, j = _nearest(p, w.float(), 5, 25.0)  # the neighbours are found from the float32 points
    full = torch.isfinite(d).all(1)
    m = p.double()[j]
    x = torch.linalg.lstsq(m, -torch.ones((len(q), 5, 1), **f8)).solution[:, :, 0]
    nrm = x.norm(dim=1, keepdim=True)
    n, dd = x / nrm, 1 / nrm[:, 0]
    e = (n[:, None] * m).sum(2) + dd[:, None]
    valid = full & (e.abs() <= 0.1).all(1)
    c = m.mean(1)
    c = c - ((n * c).sum(1) + dd)[:, None] * n
    res = torch.where(valid, (n * (w - c)).sum(1), torch.zeros_like(dd))
    planes = torch.cat([n, dd[:, None], c, torch.zeros_like(dd)[:, None]], 1) * full[:, None]
    v = (res[:, None] * n) @ R
    v = torch.where(valid[:, None], v, torch.zeros_like(v))
    gt = (res[:, None] * n * valid[:, None]).sum(0)
    go = J.T @ torch.linalg.cross(q.double(), v).sum(0)
    return dict(loss=(0.5 * res**2).sum(), grad_pose=torch.cat([go, gt]), planes=planes, res=res, valid=None, grad=v)
