"""Which frames run as one kernel and which on the queues: the last size of
one side and the first of the other for each kind of scene that the rule tells
apart, and the same image from both kernels at each. (In scenes with cones the
camera rays of one kernel are traced first, as packets: a cone's side lies
outside the box that the reference gives it, on the other side of the apex from
its base, so whether a ray finds it depends on the order of the walk.)"""
from __future__ import annotations

import dataclasses
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from pencil_b200 import _abi as A
from pencil_b200 import workloads as W
from pencil_b200.renderer import RenderSettings, RenderStats
from pencil_b200.scene import Light, Material, Scene

pytestmark = pytest.mark.gpu


def queued(st: RenderSettings) -> RenderSettings:
    return dataclasses.replace(st, block_size=128)


def kernels(name: str) -> int:
    """Launches of a frame in one kernel."""
    return 2 if name.startswith("room") else 1


def room(n: int) -> Scene:
    """A floor and n spheres, cubes, cylinders, cones and triangles of every
    material under a soft lamp (four samples), a hard lamp and a sun."""
    g = np.random.default_rng(n)
    s = Scene()
    mats = [s.add_material(Material.diffuse((0.7, 0.6, 0.5))),
            s.add_material(Material.metal((0.9, 0.8, 0.7), 0.05)),
            s.add_material(Material.dielectric(1.5))]
    s.add_plane((0, -1, 0), (0, 1, 0), mats[0])
    for k in range(n - 1):
        p, r, m = g.uniform((-5, -0.6, -2), (5, 3, 7)), float(g.uniform(0.15, 0.5)), mats[k % 3]
        axis = g.normal(size=3)
        [lambda: s.add_sphere(p, r, m), lambda: s.add_cube(p, r, m),
         lambda: s.add_cylinder(p, axis, 0.6 * r, 2 * r, m),
         lambda: s.add_cone(p, axis, r, 2 * r, m),
         lambda: s.add_triangle(p, p + g.normal(size=3) * r, p + g.normal(size=3) * r, m)][k % 5]()
    s.add_light(Light.point((6, 6, -4), (0.8, 0.8, 0.75), 0.5))
    s.add_light(Light.point((-4, 3, -3), (0.3, 0.3, 0.45), 0.0))
    s.add_light(Light.directional((0.3, -1.0, 0.4), (0.2, 0.2, 0.2)))
    s.camera = dataclasses.replace(s.camera, eye=(0.5, 1.8, -8.0), look=(0.0, 0.8, 1.0))
    return s


def matte(s: Scene) -> Scene:
    m = s.material_array().copy()
    m["kind"] = A.MAT_DIFFUSE
    s.set_material_array(m)
    return s


def lone_mesh(k: int) -> Scene:
    """The displaced icosphere without its box."""
    m = W.mesh_box(k, 64, 64).scene
    s = Scene()
    s.set_mesh(m.mesh_vertices, m.mesh_indices, s.add_material(Material.diffuse((0.7, 0.7, 0.7))))
    s.add_light(Light.point((2, 3, -3), (1, 1, 1), 0.3))
    s.camera = m.camera
    return s


SCENES = {
    "spheres": lambda: W.three_spheres_pt(64, 64).scene,
    "cloud300": lambda: W.sphere_cloud(300).scene,
    "cloud5000": lambda: W.sphere_cloud(5000).scene,
    "cloud20000": lambda: W.sphere_cloud(20_000).scene,
    "cloud40000": lambda: W.sphere_cloud(40_000).scene,
    "matte20000": lambda: matte(W.sphere_cloud(20_000).scene),
    "box338": lambda: W.mesh_box(2, 64, 64).scene,
    "lone5120": lambda: lone_mesh(4),
    "room20": lambda: room(20),
    "room123": lambda: room(123),
    "room253": lambda: room(253),
}


# (scene, path tracing, depth, samples, the largest width x height of one kernel)
LINES = [
    ("spheres", True, 4, 1, (512, 768)), ("cloud300", True, 4, 1, (1024, 512)),
    ("cloud300", True, 8, 2, (512, 512)), ("cloud5000", True, 4, 1, (512, 256)),
    ("cloud5000", True, 2, 1, (512, 256)), ("cloud5000", True, 30, 1, (1024, 512)),
    ("cloud20000", True, 4, 1, (256, 256)), ("cloud40000", True, 4, 1, (256, 192)),
    ("box338", True, 4, 1, (256, 224)), ("box338", True, 16, 1, (512, 448)),
    ("lone5120", True, 4, 2, (256, 512)), ("room20", True, 4, 1, (256, 160)),
    ("room123", True, 4, 1, (256, 88)), ("room253", True, 6, 1, (256, 132)),
    ("matte20000", False, 4, 1, (512, 512)), ("cloud300", False, 4, 1, (512, 512)),
    ("room123", False, 4, 1, (1024, 768)), ("room123", False, 3, 2, (1024, 384)),
    ("room253", False, 4, 1, (1024, 576)),
]


@pytest.mark.parametrize("name,pathtrace,depth,samples,size", LINES)
def test_both_sides_of_each_line(gpu, name, pathtrace, depth, samples, size):
    sid = gpu.upload(SCENES[name]())
    for extra in (0, 1):
        st = RenderSettings(width=size[0], height=size[1] + extra, samples=samples,
                            max_depth=depth, pathtrace=pathtrace, pathtrace_bounces=depth,
                            use_graph=False)
        stats = RenderStats()
        a = gpu.render(sid, st, stats=stats)
        assert (stats.kernel_launches == kernels(name)) == (extra == 0), stats.kernel_launches
        b = gpu.render(sid, queued(st), stats=stats)
        assert stats.kernel_launches > 2
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    gpu.free(sid)


@pytest.mark.parametrize("name", ["box338", "lone5120", "room20", "spheres", "cloud300"])
def test_frames_of_one_kernel_at_any_size(gpu, name):
    """Whitted frames of triangles, of small rooms and of matte scenes."""
    scene = SCENES[name]()
    sid = gpu.upload(matte(scene) if name == "cloud300" else scene)
    st = RenderSettings(width=1500, height=1100, samples=1, max_depth=4, use_graph=False)
    stats = RenderStats()
    a = gpu.render(sid, st, stats=stats)
    assert stats.kernel_launches == kernels(name)
    b = gpu.render(sid, queued(st))
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    gpu.free(sid)


# samples that a pixel's lanes share unevenly (9 of 8 lanes, 25 of 16)
@pytest.mark.parametrize("name,pathtrace,depth,samples,size", [
    ("spheres", True, 4, 3, (182, 120)), ("spheres", False, 3, 3, (512, 341)),
    ("box338", True, 4, 3, (64, 33)), ("room20", True, 4, 3, (64, 35)),
    ("box338", False, 3, 3, (256, 341)), ("room123", False, 2, 3, (256, 88)), ("room20", False, 2, 5, (256, 245)),
    ("matte20000", False, 4, 3, (128, 113)), ("lone5120", False, 4, 3, (128, 227)),
    ("cloud300", True, 4, 3, (256, 227)), ("room123", False, 8, 1, (1024, 1536))])
def test_lines_of_uneven_samples_and_depth(gpu, name, pathtrace, depth, samples, size):
    test_both_sides_of_each_line(gpu, name, pathtrace, depth, samples, size)


def test_cones_are_found_as_the_queues_find_them(gpu):
    """Rooms with cones in one kernel, path-traced and in Whitted mode, windows
    and second moments: the queues' image; rays of their own find other cones."""
    others = 0
    for seed in range(24):
        sid = gpu.upload(room(160 + seed))
        st = RenderSettings(width=161, height=307, samples=1 + seed % 3, max_depth=3 + seed % 5,
                            pathtrace=seed % 4 == 3, pathtrace_bounces=3, seed=seed,
                            use_graph=False)
        if st.samples == 3:
            st.height = 107
        if st.pathtrace:
            st.width, st.height, st.samples = 61, 47, 1 + seed // 4 % 2
        stats = RenderStats()
        m2 = [np.empty((st.height, st.width, 3), np.float32) for _ in range(2)]
        a = gpu.render(sid, st, None, m2[0], stats=stats)
        assert stats.kernel_launches == 2
        b = gpu.render(sid, queued(st), None, m2[1])
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), seed
        assert np.array_equal(m2[0].view(np.uint32), m2[1].view(np.uint32))
        win = (5, 7, 40, 33)
        assert np.array_equal(gpu.render_window(sid, st, win),
                              gpu.render_window(sid, queued(st), win))
        others += not np.array_equal(a, gpu.render(sid, dataclasses.replace(st, packets=False)))
        gpu.free(sid)
    assert others > 0


def cone_frames_without_room() -> None:
    import torch
    from pencil_b200.renderer import GpuContext
    from test_gpu_memory import fill
    st = RenderSettings(width=1000, height=1000, samples=1, max_depth=4, use_graph=False)
    out = torch.empty((st.height, st.width, 3), dtype=torch.float32, device="cuda")
    other = GpuContext(0)
    want = other.render(other.upload(room(60)), dataclasses.replace(st, packets=False))
    other.close()
    ctx = GpuContext(0)
    sid = ctx.upload(room(60))
    small = RenderSettings(width=32, height=32, samples=1, max_depth=4, use_graph=False)
    assert ctx.render_device(sid, small, out.data_ptr()).kernel_launches == 2
    held = fill(48 << 20)
    assert ctx.render_device(sid, st, out.data_ptr()).kernel_launches == 1
    assert np.array_equal(out.cpu().numpy().view(np.uint32), want.view(np.uint32))
    held.clear()
    torch.cuda.empty_cache()
    assert ctx.render_device(sid, small, out.data_ptr()).kernel_launches == 1
    ctx.close()
    print("done")


def test_cone_frames_without_room_for_packets():
    """A frame of cones that finds no memory for its camera rays' hits renders
    all the same, one ray per lane, and so do later ones, whose camera-relative
    nodes were given back. (In a process of its own: an allocation may also be met
    from what other contexts' pools keep.)"""
    pytest.importorskip("torch")
    here = Path(__file__).resolve().parent
    code = (f"import sys; sys.path[:0] = [{str(here)!r}, {str(here.parent)!r}]; "
            "import test_gpu_dispatch as t; t.cone_frames_without_room()")
    run = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0 and "done" in run.stdout, run.stderr[-2000:]
