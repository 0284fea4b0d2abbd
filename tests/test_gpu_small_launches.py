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
