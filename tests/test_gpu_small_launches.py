"""Launches too small to fill the GPU: the megakernel gives each pixel of a
small reference-exact image a group of lanes that share its shadow rays. The
image must be the one the ungrouped kernel makes (the ray-counting render,
which keeps one lane per pixel), bit for bit."""
from __future__ import annotations

import dataclasses

import numpy as np
import pytest

from conftest import load_golden
from pencil_b200 import _abi as A
from pencil_b200.renderer import RenderSettings
from pencil_b200.scene import Light

pytestmark = pytest.mark.gpu


# groups of 8, 4, 2 lanes and none: 148 x 32 warps hold 18,944 pixels of 8
# lanes each; the last size of each group and the first of the next
@pytest.mark.parametrize("size", [(1, 1), (64, 64), (97, 97), (18944, 1), (18945, 1), (37888, 1),
                                  (37889, 1), (75776, 1), (75777, 1), (390, 390)])
@pytest.mark.parametrize("pathtrace", [False, True])
def test_lane_groups_render_the_same_image(gpu, size, pathtrace):
    scene, _ = load_golden("prims_mix")
    sid = gpu.upload(scene)
    st = RenderSettings(width=size[0], height=size[1], samples=1, max_depth=4,
                        pathtrace=pathtrace, pathtrace_bounces=4, engine=A.ENGINE_MEGAKERNEL,
                        rng=A.RNG_PIXEL_SEQUENTIAL, glass=A.GLASS_BOTH_BRANCHES)
    a = gpu.render(sid, st)
    b = gpu.render(sid, dataclasses.replace(st, count_rays=True))
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    gpu.free(sid)


@pytest.mark.parametrize("soft", [1, 7, 40])
@pytest.mark.parametrize("binary_tree", [False, True])
def test_more_shadow_rays_than_lanes(gpu, soft, binary_tree):
    """A vertex with more shadow samples than its group has lanes takes
    several rounds; lights that are not tested and quad lights too."""
    scene, _ = load_golden("prims_mix")
    scene.add_light(Light.quad((-1, 3, -1), (1, 0, 0), (0, 0, 1), (2, 2, 2), 6))
    sid = gpu.upload(scene)
    for pathtrace in (False, True):
        st = RenderSettings(width=40, height=33, samples=2, max_depth=5, pathtrace=pathtrace,
                            pathtrace_bounces=5, soft_shadow_samples=soft,
                            engine=A.ENGINE_MEGAKERNEL, rng=A.RNG_PIXEL_SEQUENTIAL,
                            glass=A.GLASS_BOTH_BRANCHES, binary_tree=binary_tree)
        a = gpu.render(sid, st)
        b = gpu.render(sid, dataclasses.replace(st, count_rays=True))
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    gpu.free(sid)


# the last size of each group and the first of the next, by the shadow rays of a
# vertex (hard lights; 0: a light that is not tested)
@pytest.mark.parametrize("pathtrace,lights,pixels", [
    (True, 0, 64), (True, 1, 4736), (True, 2, 4736), (True, 2, 7104), (True, 3, 4736),
    (True, 6, 7104), (False, 0, 64), (False, 1, 9472), (False, 1, 37888), (False, 2, 9472),
    (False, 2, 75776), (False, 4, 37888), (False, 6, 18944), (False, 6, 75776)])
def test_lane_groups_by_shadow_rays(gpu, pathtrace, lights, pixels):
    scene, _ = load_golden("prims_mix")
    scene.lights[:] = [Light.point((0.7 * k - 2, 4, -3), (0.6, 0.5, 0.4), 0.0)
                       for k in range(max(lights, 1))]
    if lights == 0:
        scene.lights[0] = dataclasses.replace(scene.lights[0], is_emissive=True)
    sid = gpu.upload(scene)
    for n in (pixels, pixels + 1):
        st = RenderSettings(width=n, height=1, samples=1, max_depth=3, pathtrace=pathtrace,
                            pathtrace_bounces=3, engine=A.ENGINE_MEGAKERNEL,
                            rng=A.RNG_PIXEL_SEQUENTIAL, glass=A.GLASS_BOTH_BRANCHES)
        a = gpu.render(sid, st)
        b = gpu.render(sid, dataclasses.replace(st, count_rays=True))
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    gpu.free(sid)


# frames that run as one kernel unless a launch parameter asks for the queues
@pytest.mark.parametrize("name", ["three_spheres", "prims_mix", "cloud2k", "mesh_small", "shapes"])
@pytest.mark.parametrize("pathtrace", [False, True])
def test_queues_render_what_one_kernel_renders(gpu, name, pathtrace):
    """Every launch parameter that keeps a small frame on the queued kernels:
    camera packets that end their misses and compact their hits, camera rays
    one per lane, chunks, every sort key. Ragged sizes; second moments too."""
    scene, _ = load_golden(name)
    sid = gpu.upload(scene)
    for w, h, n in ((1, 1, 1), (7, 5, 2), (61, 47, 3)):
        st = RenderSettings(width=w, height=h, samples=n, max_depth=5, pathtrace=pathtrace,
                            pathtrace_bounces=5, seed=3)
        m2 = np.empty((h, w, 3), np.float32)
        ref = gpu.render(sid, st, None, m2)
        for kw in (dict(block_size=128), dict(packets=False), dict(queue_capacity=64),
                   dict(sort_key=1), dict(sort_key=2), dict(sort_key=3), dict(refill_below=1)):
            q2 = np.empty_like(m2)
            img = gpu.render(sid, dataclasses.replace(st, **kw), None, q2)
            assert np.array_equal(img.view(np.uint32), ref.view(np.uint32)), kw
            assert np.array_equal(q2.view(np.uint32), m2.view(np.uint32)), kw
    gpu.free(sid)


def test_batch_of_scenes_that_hit_and_miss(gpu):
    """Camera packets over jobs of different scenes, among them one whose
    camera sees nothing, one without primitives' light and one of depth 0."""
    from pencil_b200.scene import CameraArgs, Scene
    scene, _ = load_golden("cloud2k")
    empty = Scene()
    empty.background = (0.2, 0.3, 0.4)
    away = CameraArgs((0, 0, -120), (0, 0, -240), (0, 1, 0), 45.0, 1.0)
    sids = [gpu.upload(scene), gpu.upload(empty), gpu.upload(scene, None, away),
            gpu.upload(scene)]
    sts = [RenderSettings(width=w, height=h, samples=n, pathtrace=True, pathtrace_bounces=d)
           for w, h, n, d in ((33, 9, 1, 4), (5, 7, 2, 3), (11, 3, 3, 4), (6, 5, 1, 0))]
    outs = gpu.render_batch(sids, sts)
    for sid, st, out in zip(sids, sts, outs):
        one = gpu.render(sid, dataclasses.replace(st, packets=False))
        assert np.array_equal(out.view(np.uint32), one.view(np.uint32))
    assert np.all(outs[1] == np.array(empty.background, np.float32))
    assert not outs[3].any()
    for sid in sids:
        gpu.free(sid)


@pytest.mark.parametrize("side", [0, 1])
def test_both_sides_of_the_one_kernel_line(gpu, side):
    """A frame on the line (2^20 rays of first vertices in a small scene) and
    the next larger one: the same pixels where they are the same."""
    scene, _ = load_golden("three_spheres")
    sid = gpu.upload(scene)
    rays = 1 + sum(not l.is_emissive for l in scene.lights)
    st = RenderSettings(width=64, height=(1 << 20) // rays // 64 + side, samples=1,
                        pathtrace=True, pathtrace_bounces=3)
    a = gpu.render(sid, st)
    b = gpu.render(sid, dataclasses.replace(st, block_size=128))
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    gpu.free(sid)


@pytest.mark.parametrize("name", ["three_spheres", "prims_mix", "cloud2k", "cornell_box"])
@pytest.mark.parametrize("pathtrace", [False, True])
def test_shadow_rays_that_decide_nothing(gpu, name, pathtrace):
    """Lights behind a surface, black albedos and black lights make no shadow
    ray, except in counting renders: the same image from both, on the queues,
    in one kernel and in the reference-exact mode."""
    scene, _ = load_golden(name)
    scene.add_light(Light.point((0.3, 2.5, -3.0), (0.0, 0.0, 0.0), 0.4))
    scene.add_light(Light.directional((0.0, -1.0, 0.0), (0.4, 0.0, 0.2)))
    m = scene.material_array().copy()
    m["albedo"][0] = (0.0, 0.0, 0.0)
    scene.set_material_array(m)
    sid = gpu.upload(scene)
    st = RenderSettings(width=83, height=61, samples=2, max_depth=5, pathtrace=pathtrace,
                        pathtrace_bounces=5, seed=5)
    exact = dict(engine=A.ENGINE_MEGAKERNEL, rng=A.RNG_PIXEL_SEQUENTIAL,
                 glass=A.GLASS_BOTH_BRANCHES)
    for kw in (dict(block_size=64), dict(sort_key=3), dict(), dict(mis=True), exact):
        s = dataclasses.replace(st, **kw)
        a, b = gpu.render(sid, s), gpu.render(sid, dataclasses.replace(s, count_rays=True))
        assert np.array_equal(a, b), kw
    gpu.free(sid)


def test_automatic_capacity_over_frames_of_many_shapes(gpu):
    """One context, frames that grow the scratch by paths, then by records,
    then shrink: every image as a fresh context renders it in small chunks."""
    from pencil_b200.renderer import GpuContext
    many, _ = load_golden("prims_mix")
    for k in range(40):
        many.add_light(Light.point((0.1 * k, 4.0, -3.0), (0.02, 0.02, 0.02), 0.0))
    few, _ = load_golden("cloud2k")
    a, b = gpu.upload(few), gpu.upload(many)
    frames = [(a, few, 700, 500, 4), (b, many, 120, 90, 2), (a, few, 1200, 1100, 4),
              (b, many, 300, 200, 3), (a, few, 97, 61, 1)]
    ctx = GpuContext(0)
    ca, cb = ctx.upload(few), ctx.upload(many)
    for sid, scene, w, h, n in frames:
        st = RenderSettings(width=w, height=h, samples=n, pathtrace=True, pathtrace_bounces=3,
                            block_size=128)
        img = gpu.render(sid, st)
        ref = ctx.render(ca if sid == a else cb, dataclasses.replace(st, queue_capacity=1 << 18))
        assert np.array_equal(img.view(np.uint32), ref.view(np.uint32)), (w, h, n)
    ctx.close()
    gpu.free(a)
    gpu.free(b)


@pytest.mark.parametrize("size", [(148, 1024, 1), (151553, 1, 1), (296, 128, 2), (37889, 1, 2)])
@pytest.mark.parametrize("name,pathtrace", [("cloud2k", True), ("prims_mix", False)])
def test_register_budgets_render_the_same_image(gpu, size, name, pathtrace):
    """151,552 threads, the most that the kernel with four blocks per SM is
    launched for, and one pixel more: the counting kernel's image."""
    scene, _ = load_golden(name)
    sid = gpu.upload(scene)
    w, h, n = size
    st = RenderSettings(width=w, height=h, samples=n, max_depth=4, pathtrace=pathtrace,
                        pathtrace_bounces=4, engine=A.ENGINE_MEGAKERNEL)
    m2 = [np.empty((h, w, 3), np.float32) for _ in range(2)]
    a = gpu.render(sid, st, None, m2[0])
    b = gpu.render(sid, dataclasses.replace(st, count_rays=True), None, m2[1])
    assert np.array_equal(a, b) and np.array_equal(m2[0], m2[1])
    gpu.free(sid)


@pytest.mark.parametrize("pathtrace", [False, True])
def test_quad_lights_are_tested_whatever_their_flag(gpu, pathtrace):
    """is_emissive is the point and directional lights' way past the shadow
    test; a quad light that sets it is shadowed all the same: in the
    reference-exact groups, in one kernel, on the queues, and in gradients of
    both kinds."""
    out = []
    for flag in (False, True):
        scene, _ = load_golden("prims_mix")
        lamp = Light.quad((-1, 6, -1), (1, 0, 0), (0, 0, 1), (9, 9, 9), 1)
        scene.add_light(dataclasses.replace(lamp, is_emissive=flag))
        sid = gpu.upload(scene)
        st = RenderSettings(width=64, height=48, samples=2, max_depth=4, pathtrace=pathtrace,
                            pathtrace_bounces=4)
        exact = dict(engine=A.ENGINE_MEGAKERNEL, rng=A.RNG_PIXEL_SEQUENTIAL,
                     glass=A.GLASS_BOTH_BRANCHES)
        got = [gpu.render(sid, dataclasses.replace(st, **kw))
               for kw in (exact, dict(exact, binary_tree=True), dict(), dict(block_size=128),
                          dict(count_rays=True))]
        for w, h in ((64, 48), (300, 240)):
            dl = np.random.default_rng(1).normal(size=(h, w, 3)).astype(np.float32)
            got += gpu.adjoint(sid, dataclasses.replace(st, width=w, height=h), dl,
                               scene.n_materials, len(scene.lights), want_image=True)
        out.append(got)
        gpu.free(sid)
    for a, b in zip(*out):
        if a.dtype == np.float32:
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
        else:                       # FP64 sums in another order
            assert np.abs(a - b).max() <= 1e-9 * max(np.abs(b).max(), 1e-30)


def test_scratch_holds_frames_in_turn_not_their_product(gpu):
    """A context's scratch is the size of its largest frame: a frame of few
    paths and many records after one of many paths and one record asks for
    nothing, in either order, and nothing is given back and taken again
    between them. Images stay what they were."""
    torch = pytest.importorskip("torch")
    from pencil_b200.renderer import GpuContext
    few, _ = load_golden("three_spheres")
    some, _ = load_golden("cloud2k")
    for k in range(10):
        some.add_light(Light.point((0.1 * k, 4.0, -3.0), (0.02, 0.02, 0.02), 0.0))
    many, _ = load_golden("cloud2k")
    for k in range(70):
        many.add_light(Light.point((0.1 * k, 4.0, -3.0), (0.02, 0.02, 0.02), 0.0))
    frames = [(few, 2048, 2048, 2), (some, 141, 142, 1), (many, 120, 90, 1)]
    ctx = GpuContext(0)
    sids = [ctx.upload(f[0]) for f in frames]
    outs = [torch.empty((h, w, 3), dtype=torch.float32, device="cuda") for _, w, h, _ in frames]
    sts = [RenderSettings(width=w, height=h, samples=n, pathtrace=True, pathtrace_bounces=3,
                          block_size=128) for _, w, h, n in frames]

    def frame(k):
        ctx.render_device(sids[k], sts[k], outs[k].data_ptr())
        torch.cuda.synchronize()
        return outs[k].clone()

    first = [frame(k) for k in (1, 2, 0)]       # the largest last: nothing grows from here on
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    for k in (1, 0, 2, 1, 1, 0, 0, 2, 2):
        img = frame(k)
        assert torch.equal(img, first[(1, 2, 0).index(k)])
        # (clones come from torch's own pool)
        assert torch.cuda.mem_get_info()[0] >= free - (256 << 20), "scratch grew by the product"
        assert torch.cuda.mem_get_info()[0] <= free + (256 << 20), "scratch was given back"
    ctx.close()
