"""Host-pointer calls and the memory they are given: outputs that share memory with the
inputs (the results are those of the inputs at the beginning of the call), and the path
that copies everything (IKDG_HOST_STAGING=1) against the one that runs on the caller's
buffers, for every call that takes host inputs."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def buffer(nbytes, pinned):
    if not pinned:
        return np.zeros(nbytes, np.uint8)
    import torch
    return torch.empty(nbytes, dtype=torch.uint8, pin_memory=True).numpy()


def view(buf, at, dtype, shape):
    n = int(np.prod(shape)) * np.dtype(dtype).itemsize
    return buf[at:at + n].view(dtype).reshape(shape)


@pytest.fixture(scope="module")
def tree(ikdg_mod):
    t = ikdg_mod.KDTree()
    t.Build(np.random.default_rng(1).uniform(-10, 10, (40000, 3)).astype(np.float32))
    yield t
    t.close()


# one query a warp, eight a warp, and above the small calls' limit
@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("nq", [1, 700, 3001, 6001])
@pytest.mark.parametrize("over", ["xyz", "d2", "ids", "cnt"])
def test_knn_rows_over_the_queries(tree, nq, over, pinned):
    k = 1 if over == "xyz" else 3
    q = np.random.default_rng(nq).uniform(-10, 10, (nq, 3)).astype(np.float32)
    want = dict(zip(("ids", "d2", "xyz", "cnt"), tree.knn(q, k)))
    shape = dict(ids=(np.int32, (nq, k)), d2=(np.float32, (nq, k)), xyz=(np.float32, (nq, k, 3)), cnt=(np.int32, (nq,)))
    buf = buffer(12 * nq * 8 + 64, pinned)
    # the rows begin somewhere inside the queries' memory
    qv = view(buf, 32, np.float32, (nq, 3))
    out, at = {}, 32 + 12 * nq
    for name, (t, s) in shape.items():
        out[name] = view(buf, 32 if over == "xyz" and name == over else 32 + 4 * (nq // 2) if name == over else at, t, s)
        at += 0 if name == over else out[name].nbytes
    if over != "xyz":  # the rest of the outputs stays clear of the one that overlaps
        far = 32 + 4 * (nq // 2) + out[over].nbytes
        at = max(32 + 12 * nq, far)
        for name, (t, s) in shape.items():
            if name != over:
                out[name] = view(buf, at, t, s)
                at += out[name].nbytes
    qv[:] = q
    tree.knn_into(qv.ctypes.data, nq, k, np.inf, out["ids"].ctypes.data, out["d2"].ctypes.data, out["xyz"].ctypes.data,
                  out["cnt"].ctypes.data)
    for name in shape:
        assert np.array_equal(out[name], want[name]), name


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("nq", [1, 900, 20000])
@pytest.mark.parametrize("over", ["offsets", "ids", "xyz"])
def test_range_hits_over_the_queries(ikdg_mod, tree, nq, over, pinned):
    rng = np.random.default_rng(nq + 1)
    q = rng.uniform(-10, 10, (nq, 3)).astype(np.float32)
    r = rng.uniform(0.3, 0.6, nq).astype(np.float32)
    boxes = np.concatenate([q - r[:, None], q + r[:, None]], 1)
    for mode in ("radius", "box"):
        want = tree.radius_search(q, r) if mode == "radius" else tree.box_search(boxes)
        cap = len(want[1])
        nin = 16 * nq if mode == "radius" else 24 * nq
        sizes = dict(offsets=(np.int64, (nq + 1,)), ids=(np.int32, (cap,)), xyz=(np.float32, (cap, 3)))
        total = sum(int(np.prod(s)) * np.dtype(t).itemsize for t, s in sizes.values())
        buf = buffer(nin + total + 256, pinned)
        t, s = sizes[over]
        out = {over: view(buf, 8 * (nq // 4), t, s)}
        at = (max(nin, 8 * (nq // 4) + out[over].nbytes) + 7) // 8 * 8
        for name in ("offsets", "xyz", "ids"):
            if name != over:
                out[name] = view(buf, at, *sizes[name])
                at += out[name].nbytes
        n = C.c_int64(0)
        fp, ip, lp = C.POINTER(C.c_float), C.POINTER(C.c_int32), C.POINTER(C.c_int64)
        dst = (out["offsets"].ctypes.data_as(lp), out["ids"].ctypes.data_as(ip), out["xyz"].ctypes.data_as(fp), cap,
               C.byref(n))
        if mode == "radius":
            view(buf, 0, np.float32, (nq, 3))[:] = q
            rv = view(buf, 12 * nq, np.float32, (nq,))
            rv[:] = r
            st = tree.lib.ikdg_radius_search(tree.h, buf.ctypes.data_as(fp), nq, 3, rv.ctypes.data_as(fp), 1, *dst)
        else:
            view(buf, 0, np.float32, (nq, 6))[:] = boxes
            st = tree.lib.ikdg_box_search(tree.h, buf.ctypes.data_as(fp), nq, *dst)
        assert st == ikdg_mod.OK and n.value == cap
        for name, w in zip(("offsets", "ids", "xyz"), want):
            assert np.array_equal(out[name], w), (mode, name)


def test_copying_path_of_every_call(ikdg_mod, monkeypatch):
    rng = np.random.default_rng(9)
    direct = ikdg_mod.KDTree(0.5, 0.6, 0.4)
    monkeypatch.setenv("IKDG_HOST_STAGING", "1")
    staged = ikdg_mod.KDTree(0.5, 0.6, 0.4)
    monkeypatch.delenv("IKDG_HOST_STAGING")

    def both(f):
        a, b = f(direct), f(staged)
        for x, y in zip(*[r if isinstance(r, tuple) else (r,) for r in (a, b)]):
            assert np.array_equal(x, y)

    def state(t):
        xyz, ids = t.flatten(with_ids=True)
        o = np.argsort(ids)
        assert t.validate() == 0
        return xyz[o], ids[o], np.array([t.size(), t.validnum()]), t.tree_range()

    def hits(r):  # an insertion's points take their places in a bucket in any order
        offs, ids, xyz = r
        o = np.lexsort((ids, np.repeat(np.arange(len(offs) - 1), np.diff(offs))))
        return offs, ids[o], xyz[o]

    pts = rng.uniform(-10, 10, (30001, 3)).astype(np.float32)
    add = rng.uniform(-10, 10, (5003, 3)).astype(np.float32)
    box = rng.uniform(-10, 8, (41, 3)).astype(np.float32)
    box = np.concatenate([box, box + 1], 1)
    q = rng.uniform(-11, 11, (5001, 3)).astype(np.float32)
    steps = [lambda t: t.Build(pts), lambda t: t.Add_Points(add, True), lambda t: t.Add_Points(add[:777], False),
             lambda t: t.Delete_Points(pts[:999]), lambda t: t.Delete_Point_Boxes(box),
             lambda t: t.Add_Point_Boxes(box[:20]), lambda t: t.rebuild(),
             lambda t: t.Add_Points(rng.uniform(-10, 10, (0, 3)).astype(np.float32), True)]
    for step in steps:
        both(lambda t: np.array(step(t) or 0))
        both(state)
        for k, nq in ((1, 1), (5, 700), (9, 5001), (70, 50)):
            both(lambda t: t.knn(q[:nq], k, 3.0))
        both(lambda t: hits(t.radius_search(q[:2000], 0.7)))
        both(lambda t: hits(t.box_search(box)))
    direct.close()
    staged.close()
