"""What a user of the path-tracing core has it do, as measurable cases.

A case is one call, or the few calls, of a program that renders with this
package: a frame of a small scene, a frame of a large one, a scene loaded,
rendered once and freed, many scenes in one call, a worker's tile, a gradient
of an image loss, a tree rebuilt on the GPU, a frame turned into bytes. Scenes
are the repository's own workloads (three spheres, sphere clouds, a displaced
icosphere in a box, the box of small spheres) and a room of every primitive
kind, all generated from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from pencil_b200 import _abi as A
from pencil_b200 import workloads as W
from pencil_b200.renderer import GpuContext, RenderSettings
from pencil_b200.scene import CameraArgs, Light, Material, Scene

# Launch parameters that the autotuner settles on for large frames.
TUNED = dict(refill_below=16, sort_key=3, block_size=128)


def listed() -> list[dict]:
    return [
        # The smallest frame a user sees: the three-sphere configuration into
        # a host image, default settings. Launches and latency.
        dict(name="frame_spheres", kind="frame", scene="spheres", size=4, width=320, height=240,
             samples=2, depth=8, whitted=False, mis=False, tuned=False, host=True, lbvh=False),
        # Pencil's default mode (Whitted: soft point lights, Phong, glass) on
        # a room of every primitive kind, at an odd size, into a host image.
        dict(name="frame_whitted", kind="frame", scene="room", size=60, width=637, height=479,
             samples=2, depth=6, whitted=True, mis=False, tuned=False, host=True, lbvh=False),
        # An ordinary frame at default settings: a mid-sized cloud, ragged
        # image, nine samples, into a host image.
        dict(name="frame_cloud_20k", kind="frame", scene="cloud", size=20_000, width=641,
             height=359, samples=3, depth=8, whitted=False, mis=False, tuned=False, host=True,
             lbvh=False),
        # The headline frame: 100,000 spheres, 1280x720, 16 samples, tuned
        # launch parameters, the image left on the device.
        dict(name="frame_cloud_100k", kind="frame", scene="cloud", size=100_000, width=1280,
             height=720, samples=4, depth=8, whitted=False, mis=False, tuned=True, host=False,
             lbvh=False),
        # A triangle mesh in a box with an area light, on the traversal tree
        # the bridge picks for meshes; the largest case.
        dict(name="frame_mesh_328k", kind="frame", scene="mesh", size=7, width=1024, height=1024,
             samples=4, depth=12, whitted=False, mis=False, tuned=True, host=False, lbvh=True),
        # Pencil's --gpu call with its own tree in hand: upload, render into a
        # host image, free.
        dict(name="load_cloud_50k", kind="load", scene="cloud", size=50_000, width=960,
             height=540, samples=2, depth=8, whitted=False, mis=False, tuned=False, host=True,
             lbvh=False),
        # The same for a mesh that is looked at once (a preview, a frame of an
        # animation): loading is most of it.
        dict(name="load_mesh_82k", kind="load", scene="mesh", size=6, width=512, height=512,
             samples=1, depth=8, whitted=False, mis=False, tuned=False, host=True, lbvh=True),
        # Scenes of uneven size and resolution rendered by one call.
        dict(name="batch_32", kind="batch", size=32, samples=8, depth=8),
        # A gradient with respect to every material and light of the box of
        # 1,000 small spheres, with the image of the same samples.
        dict(name="adjoint_512", kind="adjoint", size=1000, width=512, height=512, samples=4,
             depth=6),
        # A worker's tile of a larger frame: Pencil's own random stream and
        # both glass branches, so that it equals the reference's tile.
        dict(name="tile_64", kind="tile", size=60, width=1280, height=720, samples=3, depth=6,
             tile=64),
        # Pencil's SAH tree rebuilt on the GPU for a mesh that has changed.
        dict(name="build_sah_82k", kind="build", size=6, method="sah"),
        # A 4K frame that lies on the device turned into 8-bit pixels there.
        dict(name="tonemap_4k", kind="tonemap", width=3840, height=2160, tonemap=1, exposure=0.5),
    ]


def _log(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["frame"] * 5 + ["load"] * 2 + ["batch", "adjoint", "tile", "build",
                                                       "tonemap"])
    if kind in ("frame", "load"):
        scene = rng.choice(["spheres", "room", "cloud", "cloud", "mesh"])
        if kind == "load" and scene in ("spheres", "room"):
            scene = "cloud"
        size = {"spheres": 4, "room": _log(rng, 12, 300), "cloud": _log(rng, 300, 100_000),
                "mesh": rng.randint(3, 7)}[scene]
        if kind == "load":
            size = min(size, 50_000 if scene == "cloud" else 6)
        width, height = _log(rng, 97, 1280), _log(rng, 83, 720)
        samples = rng.randint(1, 4)
        return dict(kind=kind, scene=scene, size=size, width=width, height=height,
                    samples=samples, depth=rng.randint(3, 12),
                    whitted=scene == "room" and rng.random() < 0.5,
                    mis=scene == "spheres" and rng.random() < 0.5,
                    tuned=width * height * samples * samples >= (1 << 21),
                    host=kind == "load" or rng.random() < 0.7, lbvh=scene == "mesh")
    if kind == "batch":
        return dict(kind=kind, size=rng.randint(3, 32), samples=rng.choice([1, 2, 4, 8]),
                    depth=rng.randint(3, 8))
    if kind == "adjoint":
        return dict(kind=kind, size=_log(rng, 30, 1000), width=_log(rng, 61, 512),
                    height=_log(rng, 61, 512), samples=rng.randint(1, 4),
                    depth=rng.randint(2, 6))
    if kind == "tile":
        return dict(kind=kind, size=_log(rng, 12, 300), width=_log(rng, 321, 1280),
                    height=_log(rng, 241, 720), samples=rng.randint(1, 4),
                    depth=rng.randint(2, 6), tile=rng.choice([16, 32, 61, 64]))
    if kind == "build":
        return dict(kind=kind, size=rng.randint(3, 6), method=rng.choice(["sah", "lbvh"]))
    return dict(kind=kind, width=_log(rng, 321, 3840), height=_log(rng, 239, 2160),
                tonemap=rng.randint(0, 2), exposure=round(rng.uniform(-1.0, 1.0), 3))


# ---- scenes ------------------------------------------------------------------------

def _room(n: int, seed: int) -> Scene:
    """A floor, a back wall and n primitives of every kind and material under
    a soft lamp, a hard lamp and a sun."""
    g = np.random.default_rng(seed)
    s = Scene()
    s.background = (0.1, 0.12, 0.2)
    s.ambient = (0.04, 0.04, 0.05)
    mats = [s.add_material(Material.diffuse(g.uniform(0.1, 0.9, 3), spec=0.4, shininess=24.0)),
            s.add_material(Material.diffuse(g.uniform(0.1, 0.9, 3))),
            s.add_material(Material.metal(g.uniform(0.6, 0.95, 3), 0.05)),
            s.add_material(Material.dielectric(1.5, (0.96, 0.98, 1.0)))]
    s.add_plane((0, -1, 0), (0, 1, 0), mats[0])
    s.add_quad((-8, -1, 8), (8, -1, 8), (8, 6, 8), (-8, 6, 8), mats[1])
    for k in range(n):
        p = g.uniform((-5.0, -0.6, -2.0), (5.0, 3.0, 7.0))
        r = float(g.uniform(0.15, 0.5))
        axis = g.normal(size=3)
        m = mats[int(g.integers(4))]
        kind = k % 5
        if kind == 0:
            s.add_sphere(p, r, m)
        elif kind == 1:
            s.add_cube(p, r, m)
        elif kind == 2:
            s.add_cylinder(p, axis, 0.6 * r, 2.0 * r, m)
        elif kind == 3:
            s.add_cone(p, axis, r, 2.0 * r, m)
        else:
            s.add_triangle(p, p + g.normal(size=3) * r, p + g.normal(size=3) * r, m)
    s.add_light(Light.point(g.uniform((2, 5, -5), (5, 7, -3)), (0.8, 0.8, 0.75), 0.5))
    s.add_light(Light.point(g.uniform((-5, 2, -4), (-3, 4, -2)), (0.3, 0.3, 0.45), 0.0))
    s.add_light(Light.directional((0.3, -1.0, 0.4), (0.2, 0.2, 0.2)))
    return s


def _scene(case: dict, seed: int) -> Scene:
    aspect = case["width"] / case["height"]
    if case["scene"] == "spheres":
        s = W.three_spheres_pt(case["width"], case["height"]).scene
        # another row of spheres in the same places, of the seed's own sizes
        g = np.random.default_rng(seed)
        t = Scene()
        t.background, t.ambient = s.background, s.ambient
        t.add_material_array(s.material_array())
        t.add_plane((0, 0, 0), (0, 1, 0), 0)
        for k, x in enumerate((-2.2, 0.0, 2.2)):
            r = float(g.uniform(0.8, 1.05))
            t.add_sphere((x, r, float(g.uniform(-0.3, 0.3))), r, k + 1)
        t.add_light(s.lights[0])
        t.camera = s.camera
        return t
    if case["scene"] == "room":
        s = _room(case["size"], seed)
        s.camera = CameraArgs((0.5, 1.8, -8.0), (0.0, 0.8, 1.0), (0, 1, 0), 55.0, aspect)
        return s
    if case["scene"] == "cloud":
        return W.sphere_cloud(case["size"], case["width"], case["height"], seed=seed).scene
    return W.mesh_box(case["size"], case["width"], case["height"], seed=seed).scene


def _settings(case: dict, seed: int) -> RenderSettings:
    st = RenderSettings(width=case["width"], height=case["height"], samples=case["samples"],
                        max_depth=case["depth"], pathtrace=not case.get("whitted", False),
                        pathtrace_bounces=case["depth"], mis=case.get("mis", False),
                        seed=seed & 0xFFFF)
    if case.get("tuned"):
        paths = case["width"] * case["height"] * case["samples"] ** 2
        st.queue_capacity = min(1 << 24, 1 << max(0, paths - 1).bit_length())
        for k, v in TUNED.items():
            setattr(st, k, v)
    return st


# ---- the cases ---------------------------------------------------------------------

def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    ctx = GpuContext(0)
    state = dict(case=case, ctx=ctx)
    if kind in ("frame", "load"):
        scene = _scene(case, seed)
        if case["lbvh"]:
            ctx.set_traversal_tree(A.TRAVERSAL_LBVH)
        nodes, _ = scene.build_bvh()
        state.update(scene=scene, nodes=nodes, st=_settings(case, seed))
        if kind == "frame":
            state["sid"] = ctx.upload(scene, nodes)
        shape = (case["height"], case["width"], 3)
        state["out"] = (np.empty(shape, np.float32) if case["host"]
                        else torch.empty(shape, dtype=torch.float32, device="cuda"))
    elif kind == "batch":
        # the jobs' sizes are the case's, their scenes the seed's
        g = np.random.default_rng(case["size"])
        sids, sts, outs = [], [], []
        for k in range(case["size"]):
            n = int(np.exp(g.uniform(np.log(10), np.log(50_000))))
            res = int(g.choice([128, 256, 512]))
            samples = int(g.choice([v for v in (1, 2, 4, 8) if v <= case["samples"]]))
            w = W.sphere_cloud(n, res, res, samples, case["depth"], seed=seed * 1000 + k)
            w.settings.seed = k
            nodes, _ = w.scene.build_bvh()
            sids.append(ctx.upload(w.scene, nodes))
            sts.append(w.settings)
            outs.append(torch.empty((res, res, 3), dtype=torch.float32, device="cuda"))
        state.update(sids=sids, sts=sts, outs=outs, ptrs=[o.data_ptr() for o in outs])
    elif kind == "adjoint":
        w, _, _ = W.adjoint_box(case["size"], case["width"], case["height"], case["samples"],
                                case["depth"], seed=seed)
        w.settings.seed = seed & 0xFFFF
        g = np.random.default_rng(seed)
        dl = g.normal(0.5, 1.0, size=(case["height"], case["width"], 3)).astype(np.float32)
        state.update(sid=ctx.upload(w.scene), st=w.settings, dl=dl, n_mat=w.scene.n_materials,
                     n_light=len(w.scene.lights))
    elif kind == "tile":
        scene = _room(case["size"], seed)
        scene.camera = CameraArgs((0.5, 1.8, -8.0), (0.0, 0.8, 1.0), (0, 1, 0), 55.0,
                                  case["width"] / case["height"])
        st = RenderSettings(width=case["width"], height=case["height"], samples=case["samples"],
                            max_depth=case["depth"], rng=A.RNG_PIXEL_SEQUENTIAL,
                            glass=A.GLASS_BOTH_BRANCHES, engine=A.ENGINE_MEGAKERNEL)
        # a tile off the middle of the frame, where the primitives are
        x, y = case["width"] // 2 - case["tile"] // 3, case["height"] // 2 - case["tile"] // 4
        state.update(sid=ctx.upload(scene), st=st, xy=(x, y))
    elif kind == "build":
        state["scene"] = W.mesh_box(case["size"], seed=seed).scene
    else:
        g = torch.Generator(device="cuda").manual_seed(seed)
        shape = (case["height"], case["width"], 3)
        # a rendered frame's range: mostly below 1, a few highlights above
        state["hdr"] = torch.rand(shape, generator=g, device="cuda") ** 2 / (
            torch.rand(shape, generator=g, device="cuda") + 0.05)
        state["rgb8"] = torch.empty(shape, dtype=torch.uint8, device="cuda")
    return state


def run(state: dict):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "frame":
        if case["host"]:
            return ctx.render(state["sid"], state["st"], state["out"])
        ctx.render_device(state["sid"], state["st"], state["out"].data_ptr())
        return state["out"]
    if kind == "load":
        sid = ctx.upload(state["scene"], state["nodes"])
        ctx.render(sid, state["st"], state["out"])
        ctx.free(sid)
        return state["out"]
    if kind == "batch":
        ctx.render_batch(state["sids"], state["sts"], device_ptrs=state["ptrs"])
        return state["outs"]
    if kind == "adjoint":
        da, de, dl, img = ctx.adjoint(state["sid"], state["st"], state["dl"], state["n_mat"],
                                      state["n_light"], want_image=True)
        # the parameters a program optimises are float32, and so are its gradients
        return dict(d_albedo=da.astype(np.float32), d_emission=de.astype(np.float32),
                    d_light=dl.astype(np.float32), image=img)
    if kind == "tile":
        return ctx.render_tile(state["sid"], state["st"], *state["xy"], case["tile"],
                               case["tile"])
    if kind == "build":
        nodes, depth = ctx.build_bvh_device(state["scene"], case["method"])
        return dict(bmin=nodes["bmin"], bmax=nodes["bmax"], left=nodes["left"],
                    right=nodes["right"], depth=depth)
    hdr, rgb8 = state["hdr"], state["rgb8"]
    ctx.check(ctx.lib.pgpu_tonemap(ctx.h, hdr.data_ptr(), hdr.numel() // 3, case["tonemap"],
                                   float(case["exposure"]),
                                   A.TONEMAP_DEVICE_INPUT | A.TONEMAP_DEVICE_OUTPUT,
                                   rgb8.data_ptr()), "pgpu_tonemap")
    return rgb8


def _rays(paths: float, depth: int, n: int) -> float:
    """Operations of `paths` paths in a scene of n primitives, at the least:
    two rays per bounce over half the depth, each going down one root-to-leaf
    path of a 4-wide tree (24 operations a box) to one primitive test."""
    levels = max(1.0, math.log(max(n, 2), 4))
    return paths * max(1.0, depth / 2) * 2 * (levels * 4 * 24 + 60)


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("frame", "load"):
        n = 20 * 4 ** case["size"] if case["scene"] == "mesh" else case["size"]
        pixels = case["width"] * case["height"]
        scene = n * (64 + 48 + 64)      # a wide node's share, geometry, material
        if kind == "load":
            scene += n * (64 + 2 * 32)  # the caller's primitives and tree
        return dict(bytes=scene + 12 * pixels,
                    flops=_rays(pixels * case["samples"] ** 2, case["depth"], n))
    if kind == "batch":
        # the mean job: 114,688 pixels (of 128, 256 and 512 squared)
        spp = [v * v for v in (1, 2, 4, 8) if v <= case["samples"]]
        paths = case["size"] * 114_688 * sum(spp) / len(spp)
        return dict(bytes=case["size"] * (114_688 * 12 + 5_900 * 176),
                    flops=_rays(paths, case["depth"], 5_900))
    if kind == "adjoint":
        pixels = case["width"] * case["height"]
        return dict(bytes=24 * pixels + case["size"] * (176 + 48),
                    flops=1.5 * _rays(pixels * case["samples"] ** 2, case["depth"], case["size"]))
    if kind == "tile":
        pixels = case["tile"] ** 2
        return dict(bytes=12 * pixels + case["size"] * 176,
                    flops=_rays(pixels * case["samples"] ** 2, 2 * case["depth"], case["size"]))
    if kind == "build":
        n = 20 * 4 ** case["size"]
        return dict(bytes=n * (12 + 6) + n * 64, flops=n * math.log2(n) * 12)
    return dict(bytes=case["width"] * case["height"] * 15, flops=case["width"] * case["height"] * 60)


def exact(case: dict, seed: int):
    """No case has a 64-bit value: a path in 64 bits rounds to other hits and
    other roulette decisions than the same path in 32, so it is another
    estimate of the picture, not a more exact one; a tree's boxes and a
    frame's bytes are selections, equal or not."""
    return None
