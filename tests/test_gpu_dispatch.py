"""Which frames run as one kernel and which on the queues: the last size of
one side and the first of the other for each kind of scene that the rule tells
apart, and the same image from both kernels at each. (Rooms against the queues
without camera packets: a cone's side lies outside the box that the reference
gives it, on the other side of the apex from its base, so whether a ray finds
it depends on the order of the walk, and packets take another.)"""
from __future__ import annotations

import dataclasses

import numpy as np
import pytest

from pencil_b200 import _abi as A
from pencil_b200 import workloads as W
from pencil_b200.renderer import RenderSettings, RenderStats
from pencil_b200.scene import Light, Material, Scene

pytestmark = pytest.mark.gpu


def queued(name: str, st: RenderSettings) -> RenderSettings:
    return dataclasses.replace(st, **(dict(packets=False) if name.startswith("room")
                                      else dict(block_size=128)))


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
        assert (stats.kernel_launches == 1) == (extra == 0), stats.kernel_launches
        b = gpu.render(sid, queued(name if extra == 0 else "", st), stats=stats)
        assert stats.kernel_launches > 1
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
    assert stats.kernel_launches == 1
    b = gpu.render(sid, queued(name, st))
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    gpu.free(sid)


# samples that a pixel's lanes share unevenly (9 of 8 lanes, 25 of 16)
@pytest.mark.parametrize("name,pathtrace,depth,samples,size", [
    ("spheres", True, 4, 3, (182, 120)), ("spheres", False, 3, 3, (512, 341)),
    ("box338", True, 4, 3, (64, 24)), ("box338", False, 3, 3, (256, 341)),
    ("room123", False, 2, 3, (256, 88)), ("room20", False, 2, 5, (256, 81)),
    ("matte20000", False, 4, 3, (128, 113)), ("lone5120", False, 4, 3, (128, 227)),
    ("cloud300", True, 4, 3, (256, 227))])
def test_lines_of_uneven_samples(gpu, name, pathtrace, depth, samples, size):
    test_both_sides_of_each_line(gpu, name, pathtrace, depth, samples, size)
