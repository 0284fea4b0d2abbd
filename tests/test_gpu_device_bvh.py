"""pgpu_build_bvh_device: a linear BVH built on the GPU in Pencil's node-table
format. It is a different tree from Pencil's SAH tree, so the checks are on
its structure and on what it finds: a valid DFS pre-order table with every
primitive in one leaf (the upload validates it too), the same closest-hit
distances as Pencil's tree for camera and random rays (the primitive may
differ only between surfaces at exactly the same distance), and renders
that agree with those on Pencil's tree."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import GOLDEN_SCENES, load_golden
from pencil_b200 import _abi as A
from pencil_b200 import workloads as W
from pencil_b200.renderer import RenderSettings

pytestmark = pytest.mark.gpu


def check_table(nodes: np.ndarray, n_prims: int) -> int:
    """Validates DFS pre-order links and leaves; returns the depth."""
    assert len(nodes) == max(2 * n_prims - 1, 0)
    if n_prims == 0:
        return 0
    size = np.zeros(len(nodes), np.int64)
    for k in range(len(nodes) - 1, -1, -1):
        nd = nodes[k]
        if nd["left"] < 0:
            size[k] = 1
            continue
        assert nd["left"] == k + 1 and nd["right"] == nd["left"] + size[nd["left"]]
        size[k] = 1 + size[nd["left"]] + size[nd["right"]]
        for c in (nd["left"], nd["right"]):        # parent box holds the child's
            assert np.all(nodes[c]["bmin"] >= nd["bmin"]) and np.all(nodes[c]["bmax"] <= nd["bmax"])
    assert size[0] == len(nodes)
    leaves = nodes[nodes["left"] < 0]["right"]
    assert sorted(leaves.tolist()) == list(range(n_prims))
    level = np.zeros(len(nodes), np.int64)
    level[0] = 1
    for k in range(len(nodes)):
        if nodes[k]["left"] >= 0:
            level[nodes[k]["left"]] = level[nodes[k]["right"]] = level[k] + 1
    return int(level.max())


@pytest.mark.parametrize("name", GOLDEN_SCENES)
def test_device_tree_is_valid_and_finds_the_same_hits(gpu, name):
    scene, fx = load_golden(name)
    nodes, depth = gpu.build_bvh_device(scene)
    assert check_table(nodes, scene.n_unified) == depth
    sid_host = gpu.upload(scene, fx["nodes"])
    sid_dev = gpu.upload(scene, nodes)
    rng = np.random.default_rng(5)
    uv = rng.uniform(0, 1, (20000, 2)).astype(np.float32)
    ph, th = gpu.primary_hits(sid_host, uv)
    pd, td = gpu.primary_hits(sid_dev, uv)
    assert np.array_equal(th.view(np.uint32), td.view(np.uint32))
    assert (ph == pd).mean() >= 0.999          # ties at equal distance may pick another
    ph, th = gpu.trace_rays(sid_host, fx["rays"])
    pd, td = gpu.trace_rays(sid_dev, fx["rays"])
    assert np.array_equal(th.view(np.uint32), td.view(np.uint32))
    assert (ph == pd).mean() >= 0.999
    gpu.free(sid_host)
    gpu.free(sid_dev)


def test_device_tree_edge_cases(gpu):
    from pencil_b200.scene import Material, Scene
    s = Scene()
    assert len(gpu.build_bvh_device(s)[0]) == 0
    m = s.add_material(Material.diffuse((0.5, 0.5, 0.5)))
    s.add_sphere((0, 0, 0), 1.0, m)
    nodes, depth = gpu.build_bvh_device(s)
    assert len(nodes) == 1 and depth == 1
    for _ in range(40):                         # identical centres: keys tie on Morton code
        s.add_sphere((1.0, 2.0, 3.0), 0.5, m)
    nodes, depth = gpu.build_bvh_device(s)
    assert check_table(nodes, s.n_unified) == depth


def test_device_tree_renders_the_sphere_cloud_and_the_mesh(gpu):
    for wl, size in ((W.sphere_cloud(), (320, 180)), (W.mesh_box(subdiv=5), (128, 128))):
        st = wl.settings
        st.width, st.height = size
        st.samples = 2
        nodes, depth = gpu.build_bvh_device(wl.scene)
        assert check_table(nodes, wl.scene.n_unified) == depth
        a = gpu.upload(wl.scene)
        b = gpu.upload(wl.scene, nodes)
        ia, ib = gpu.render(a, st), gpu.render(b, st)
        same = np.all(ia.view(np.uint32) == ib.view(np.uint32), axis=2).mean()
        assert same >= 0.999, same
        gpu.free(a)
        gpu.free(b)


# ---- Pencil's SAH tree built on the device (pgpu_build_bvh_device_sah) ----------------
@pytest.mark.parametrize("name", GOLDEN_SCENES)
def test_device_sah_tree_valid_and_hits_equal(gpu, name):
    """Valid table; the same hits as the reference's tree; node for node the
    reference's tree except where a median split meets tied centroid keys."""
    scene, fx = load_golden(name)
    nodes, depth = gpu.build_bvh_device(scene, method="sah")
    assert check_table(nodes, scene.n_unified) == depth
    same = np.mean([a.tobytes() == b.tobytes() for a, b in zip(nodes, fx["nodes"])])
    print(f"{name}: {same:.4f} of nodes equal to the reference tree's")
    sid_host = gpu.upload(scene, fx["nodes"])
    sid_dev = gpu.upload(scene, nodes)
    ph, th = gpu.trace_rays(sid_host, fx["rays"])
    pd, td = gpu.trace_rays(sid_dev, fx["rays"])
    assert np.array_equal(th.view(np.uint32), td.view(np.uint32))
    assert (ph == pd).mean() >= 0.999
    gpu.free(sid_host)
    gpu.free(sid_dev)


@pytest.mark.parametrize("wl_name", ["sphere_cloud", "cloud_seed3", "sphere_batch"])
def test_device_sah_equals_reference_tree_without_ties(gpu, wl_name):
    """Random sphere scenes have no tied centroid keys: the device build is
    Pencil's SAH tree node for node (the host build equals the reference's,
    test_oracle_golden.py / test_oracle_config_pins.py)."""
    import time
    if wl_name == "sphere_cloud":
        scene = W.sphere_cloud().scene
    elif wl_name == "cloud_seed3":
        scene = W.sphere_cloud(20000, 64, 64, 1, 8, seed=3).scene
    else:
        scene = W.sphere_batch(n_scenes=3, seed=8)[2].scene
    t0 = time.perf_counter()
    host, hdepth = scene.build_bvh()
    t1 = time.perf_counter()
    gpu.build_bvh_device(scene, method="sah")
    t2 = time.perf_counter()
    dev, ddepth = gpu.build_bvh_device(scene, method="sah")
    t3 = time.perf_counter()
    print(f"{wl_name}: {scene.n_unified} primitives, host SAH {1e3 * (t1 - t0):.1f} ms, "
          f"device SAH {1e3 * (t3 - t2):.1f} ms")
    assert ddepth == hdepth
    assert dev.tobytes() == host.tobytes()


def test_device_sah_on_the_full_mesh(gpu):
    """The 1,310,720-triangle mesh box: symmetric triangles tie in median
    splits, so the trees differ in places; the table is valid, its depth is
    the host tree's give or take, and it finds the same hit distances (and,
    but for surfaces at exactly equal distances, the same primitives)."""
    import time
    w = W.mesh_box()
    host, hdepth = w.scene.build_bvh()
    gpu.build_bvh_device(w.scene, method="sah")
    t0 = time.perf_counter()
    dev, ddepth = gpu.build_bvh_device(w.scene, method="sah")
    ms = 1e3 * (time.perf_counter() - t0)
    same = np.mean(dev["left"] == host["left"])
    print(f"mesh: device SAH {ms:.1f} ms, depth {ddepth} (host {hdepth}), "
          f"{same:.4f} of nodes with the host tree's shape")
    assert check_table(dev, w.scene.n_unified) == ddepth
    assert abs(ddepth - hdepth) <= 4
    sa, sb = gpu.upload(w.scene, host), gpu.upload(w.scene, dev)
    uv = np.random.default_rng(9).uniform(0, 1, (50000, 2)).astype(np.float32)
    pa, ta = gpu.primary_hits(sa, uv)
    pb, tb = gpu.primary_hits(sb, uv)
    assert np.array_equal(ta.view(np.uint32), tb.view(np.uint32))
    assert (pa == pb).mean() >= 0.999
    gpu.free(sa)
    gpu.free(sb)


def test_device_sah_edge_cases(gpu):
    from pencil_b200.scene import Material, Scene
    s = Scene()
    assert len(gpu.build_bvh_device(s, method="sah")[0]) == 0
    m = s.add_material(Material.diffuse((0.5, 0.5, 0.5)))
    s.add_sphere((0, 0, 0), 1.0, m)
    assert len(gpu.build_bvh_device(s, method="sah")[0]) == 1
    for k in range(3):                          # 2 to 4 primitives: the root is small
        s.add_sphere((k + 1.0, 0.5 * k, 0), 0.5, m)
        nodes, depth = gpu.build_bvh_device(s, method="sah")
        host, hdepth = s.build_bvh()
        assert nodes.tobytes() == host.tobytes() and depth == hdepth
    for _ in range(40):                         # identical boxes: every split is a median split
        s.add_sphere((1.0, 2.0, 3.0), 0.5, m)
    nodes, depth = gpu.build_bvh_device(s, method="sah")
    assert check_table(nodes, s.n_unified) == depth
    s.add_plane((0, -1, 0), (0, 1, 0), m)       # a +-1e6 box: the root's bins all fall together
    nodes, depth = gpu.build_bvh_device(s, method="sah")
    assert check_table(nodes, s.n_unified) == depth


@pytest.mark.parametrize("n", [5, 6, 31, 33, 511, 512, 513, 514, 1026, 1537, 5000])
@pytest.mark.parametrize("kind", ["random", "grid", "line", "point", "lopsided"])
def test_device_sah_subtrees_built_by_one_block(gpu, n, kind):
    """Sizes around the subtrees that one block builds (512), with centres
    that spread, tie, lie on a line, coincide (median splits only) or crowd
    (deep trees): a valid table, and where no centre ties Pencil's tree node
    for node."""
    from pencil_b200.scene import Material, Scene
    rng = np.random.default_rng(n)
    c = rng.uniform(-10, 10, (n, 3)).astype(np.float32)
    if kind == "grid":
        c = np.round(c)
    elif kind == "line":
        c[:, 1:] = 0
    elif kind == "point":
        c[:] = c[0]
    elif kind == "lopsided":
        c = (np.sign(c) * np.abs(c / 10) ** 9 * 1e4).astype(np.float32)
    s = Scene()
    m = s.add_material(Material.diffuse((1, 1, 1)))
    s.add_spheres(c, rng.uniform(0.01, 0.3, n).astype(np.float32), np.full(n, m, np.int32))
    nodes, depth = gpu.build_bvh_device(s, "sah")
    assert check_table(nodes, n) == depth
    if kind == "random":
        host, host_depth = s.build_bvh()
        assert depth == host_depth and np.array_equal(nodes, host)


# ---- primitives that are not finite ------------------------------------------------
# pgpu_build_bvh_device* take any bits (an upload does not): the table must
# still hold every primitive once.

def _ord(f):
    """The int image that orders floats as their bits do; NaN as the device makes it."""
    i = np.where(np.isnan(f), np.int32(0x7fffffff), np.asarray(f, np.float32).view(np.int32))
    return np.where(i >= 0, i, i ^ np.int32(0x7fffffff)).astype(np.int32)


def _unord(i):
    i = np.asarray(i, np.int32)
    return np.where(i >= 0, i, i ^ np.int32(0x7fffffff)).astype(np.int32).view(np.float32)


def _ord_box(mn, mx):
    """Bounds of boxes by bit order: a NaN plane is the largest."""
    return (_unord(np.minimum(_ord(mn).min(0), _ord(np.float32(1e30)))),
            _unord(np.maximum(_ord(mx).max(0), _ord(np.float32(-1e30)))))


def _axis(mn, mx):
    e = mx - mn
    return 0 if e[0] >= e[1] and e[0] >= e[2] else 1 if e[1] >= e[2] else 2


def _area(mn, mx):
    e = mx - mn
    return np.float32(2) * (e[0] * e[1] + e[1] * e[2] + e[0] * e[2])


def sah_model(mn, mx):
    """The device's SAH build over boxes of any bits, one node at a time."""
    F = np.float32
    n = len(mn)
    out = np.zeros(2 * n - 1, A.NODE_DTYPE)
    empty = (np.full(3, 1e30, F), np.full(3, -1e30, F))

    def write(at, box, left, right):
        out[at] = (box[0], left, box[1], right)

    def small(items, node):
        lo, hi = (np.fmin.reduce(np.vstack([empty[0][None], mn[items]])),
                  np.fmax.reduce(np.vstack([empty[1][None], mx[items]])))
        if len(items) == 1:
            return write(node, (lo, hi), -1, items[0])
        a = _axis(lo, hi)
        items = list(items)
        for i in range(1, len(items)):
            v, j = items[i], i - 1
            while j >= 0 and mn[items[j], a] + mx[items[j], a] > mn[v, a] + mx[v, a]:
                items[j + 1] = items[j]
                j -= 1
            items[j + 1] = v
        h = len(items) // 2
        write(node, (lo, hi), node + 1, node + 2 * h)
        small(items[:h], node + 1)
        small(items[h:], node + 2 * h)

    def build(items, node, box):
        if len(items) == 1:
            return write(node, box, -1, items[0])
        if len(items) <= 4:
            return small(items, node)
        a = _axis(*box)
        best, cut, sides = np.finfo(F).max, 0, None
        if box[1][a] > box[0][a]:
            f = ((mn[items, a] + mx[items, a]) * F(0.5) - box[0][a]) / (box[1][a] - box[0][a]) * F(12)
            k = np.nan_to_num(f, nan=0.0, posinf=12.0, neginf=0.0).clip(0, 11).astype(int)
            bins = [_ord_box(mn[items[k == q]], mx[items[k == q]]) if (k == q).any() else empty
                    for q in range(12)]
            sa = _area(*box)
            for b in range(1, 12):
                nl = int((k < b).sum())
                if nl == 0 or nl == len(items):
                    continue
                half = [(np.fmin.reduce([empty[0]] + [x[0] for x in part]),
                         np.fmax.reduce([empty[1]] + [x[1] for x in part]))
                        for part in (bins[:b], bins[b:])]
                cost = F(1) + (F(nl) * _area(*half[0]) + F(len(items) - nl) * _area(*half[1])) / \
                    (sa if sa > 0 else F(1))
                if cost < best:
                    best, cut, sides = cost, b, half
        if cut:
            left, right = items[k < cut], items[k >= cut]
        else:
            order = items[np.argsort(_ord(mn[items, a] + mx[items, a] + F(0)), kind="stable")]
            left, right = order[:len(items) // 2], order[len(items) // 2:]
            sides = [_ord_box(mn[p], mx[p]) for p in (left, right)]
        write(node, box, node + 1, node + 2 * len(left))
        build(left, node + 1, sides[0])
        build(right, node + 2 * len(left), sides[1])

    with np.errstate(all="ignore"):
        if n > 4:
            build(np.arange(n), 0, (_unord(_ord(mn).min(0)), _unord(_ord(mx).max(0))))
        else:
            small(np.arange(n), 0)
    return out


def leaves_once(nodes, n):
    """Links of a DFS table, and every primitive in one leaf (boxes aside)."""
    plain = nodes.copy()
    plain["bmin"], plain["bmax"] = 0, 0
    return check_table(plain, n)


@pytest.mark.parametrize("n", [5, 7, 33, 512, 513, 1500])
@pytest.mark.parametrize("kind", ["nan", "nan_axis", "inf", "all_nan", "half_nan_point"])
def test_device_builds_of_primitives_that_are_not_finite(gpu, n, kind):
    from pencil_b200.scene import Material, Scene
    rng = np.random.default_rng(n)
    c = rng.uniform(-10, 10, (n, 3)).astype(np.float32)
    r = rng.uniform(0.01, 0.3, n).astype(np.float32)
    if kind == "nan":
        c[rng.choice(n, max(n // 10, 1), replace=False)] = np.nan
    elif kind == "nan_axis":
        for a in range(3):
            c[rng.choice(n, max(n // 20, 1), replace=False), a] = np.nan
    elif kind == "inf":
        r[rng.choice(n, max(n // 10, 1), replace=False)] = np.inf
        c[0] = (-np.inf, np.inf, 0)
    elif kind == "all_nan":
        c[:] = np.nan
    else:
        c[:] = c[0]
        c[::2] = np.nan
    s = Scene()
    m = s.add_material(Material.diffuse((1, 1, 1)))
    s.add_spheres(c, r, np.full(n, m, np.int32))
    nodes, depth = gpu.build_bvh_device(s, "sah")
    assert leaves_once(nodes, n) == depth
    with np.errstate(all="ignore"):
        want = sah_model(c - r[:, None], c + r[:, None])
    assert np.array_equal(nodes["left"], want["left"])
    assert np.array_equal(nodes["right"], want["right"])
    assert np.array_equal(nodes["bmin"], want["bmin"], equal_nan=True)
    assert np.array_equal(nodes["bmax"], want["bmax"], equal_nan=True)
    nodes, depth = gpu.build_bvh_device(s, "lbvh")
    assert leaves_once(nodes, n) == depth


def test_device_builds_of_a_mesh_with_broken_vertices(gpu):
    w = W.mesh_box(4, 8, 8, 1, 1)
    s, rng = w.scene, np.random.default_rng(3)
    v = s.mesh_vertices.copy()
    v[rng.choice(len(v), len(v) // 20, replace=False)] = np.nan
    v[rng.choice(len(v), len(v) // 20, replace=False), 1] = np.inf
    s.set_mesh(v, s.mesh_indices, s.mesh_materials)
    for method in ("sah", "lbvh"):
        nodes, depth = gpu.build_bvh_device(s, method)
        assert leaves_once(nodes, s.n_unified) == depth
