"""Small frames on the queued kernels: the wavefront engine renders them as one
kernel unless a launch parameter is set, so the tests of small frames in
test_gpu_parity.py run here once more with one set, and frame graphs, which
only the queues use, are followed over scenes."""
from __future__ import annotations

import dataclasses

import numpy as np
import pytest

import test_gpu_parity as P
from conftest import GOLDEN_SCENES
from pencil_b200 import _abi as A
from pencil_b200 import workloads as W
from pencil_b200.renderer import GpuContext, RenderStats
from test_gpu_parity import scenes  # noqa: F401 (a fixture)

pytestmark = pytest.mark.gpu


class Queued:
    """The context with every wavefront frame on the queues."""

    def __init__(self, ctx):
        self.ctx = ctx
        self.frames = 0

    def __getattr__(self, name):
        return getattr(self.ctx, name)

    def _settings(self, st):
        if st.engine != A.ENGINE_WAVEFRONT:
            return st
        self.frames += 1
        return dataclasses.replace(st, block_size=128)

    def render(self, sid, st, *args, **kw):
        q = self._settings(st)
        if q is not st and not st.count_rays:
            stats = RenderStats()
            img = self.ctx.render(sid, dataclasses.replace(q, use_graph=False), stats=stats)
            assert stats.kernel_launches > 1
            assert np.array_equal(self.ctx.render(sid, q, *args, **kw), img)
            return img
        return self.ctx.render(sid, q, *args, **kw)

    def render_window(self, sid, st, *args, **kw):
        return self.ctx.render_window(sid, self._settings(st), *args, **kw)


@pytest.fixture
def queued(gpu):
    q = Queued(gpu)
    yield q
    assert q.frames > 0


@pytest.mark.parametrize("name", GOLDEN_SCENES)
@pytest.mark.parametrize("mode", ["pt", "wh"])
def test_production_estimator_matches_oracle(queued, scenes, name, mode):  # noqa: F811
    P.test_production_estimator_matches_oracle_path_for_path(queued, scenes, name, mode)


@pytest.mark.parametrize("seed", [15, 16, 17])
def test_mis_path_tracing(queued, seed):
    P.test_mis_path_tracing(queued, seed)


def test_quad_light_box_matches_oracle(queued):
    P.test_quad_light_box_matches_oracle(queued)


def test_edge_cases(queued):
    P.test_edge_cases(queued)


def test_renders_are_deterministic(queued, scenes):  # noqa: F811
    P.test_renders_are_deterministic(queued, scenes)


def test_window_render_equals_the_crop(queued, scenes):  # noqa: F811
    P.test_window_render_equals_the_crop_of_the_frame(queued, scenes, A.ENGINE_WAVEFRONT)


def test_frame_graph_follows_the_scene():
    """Frames of one shape replay one graph, updated for each scene: two scenes
    in turn, then a third in the freed first one's place, whose nodes (and
    nodes relative to the camera) may lie where the first one's lay."""
    ctx = GpuContext(0)
    jobs = W.sphere_batch(n_scenes=3, seed=23)
    st = dataclasses.replace(jobs[0].settings, width=80, height=64, block_size=128)
    want = []
    for j in jobs:
        sid = ctx.upload(j.scene)
        want.append(ctx.render(sid, dataclasses.replace(st, use_graph=False)))
        ctx.free(sid)
    a, b = ctx.upload(jobs[0].scene), ctx.upload(jobs[1].scene)
    stats = RenderStats()
    launches = []
    for sid, k in ((a, 0), (a, 0), (a, 0), (b, 1), (a, 0), (b, 1), (b, 1)):
        img = ctx.render(sid, st, stats=stats)
        launches.append(stats.kernel_launches)
        assert np.array_equal(img.view(np.uint32), want[k].view(np.uint32))
    assert launches[2:] == [1] * 5, launches          # graphs
    ctx.free(a)
    c = ctx.upload(jobs[2].scene)
    for sid, k in ((c, 2), (b, 1), (c, 2)):
        img = ctx.render(sid, st, stats=stats)
        assert stats.kernel_launches == 1
        assert np.array_equal(img.view(np.uint32), want[k].view(np.uint32))
    ctx.close()
