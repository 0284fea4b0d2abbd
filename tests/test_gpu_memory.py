"""Calls that find the device's memory taken by what the context keeps to be
fast (the renders' scratch, camera-relative nodes) get it instead: uploads,
device tree builds and renders that would fit without it succeed."""
from __future__ import annotations

import numpy as np
import pytest

from pencil_b200 import _abi as A
from pencil_b200 import workloads as W
from pencil_b200.renderer import GpuContext, RenderSettings

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def fill(leave: int) -> list:
    """Takes the device's free memory but for `leave` bytes."""
    held = []
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    while (room := torch.cuda.mem_get_info()[0] - leave) >= 4 << 20:
        held.append(torch.empty(min(room, 16 << 30) & ~0x1fffff, dtype=torch.uint8, device="cuda"))
    return held


def big_frame(ctx, sid) -> None:
    """2^24 paths on the queues: about 4.6 GB of scratch."""
    st = RenderSettings(width=4096, height=4096, samples=1, pathtrace=True, pathtrace_bounces=2,
                        block_size=128)
    out = torch.empty((st.height, st.width, 3), dtype=torch.float32, device="cuda")
    ctx.render_device(sid, st, out.data_ptr())
    torch.cuda.synchronize()


@pytest.fixture
def full():
    """A context with scratch and warm kernels, in a device with 48 MiB left
    (less than any of the calls below takes)."""
    scene = W.sphere_cloud(600_000).scene
    other = GpuContext(0)           # (its pool keeps what the build takes)
    nodes, depth = other.build_bvh_device(scene, "lbvh")
    other.close()
    ctx = GpuContext(0)
    warm = W.mesh_box(3, 64, 64, 1, 2)
    for tree in (A.TRAVERSAL_LBVH, A.TRAVERSAL_SAH, A.TRAVERSAL_UPLOADED):
        ctx.set_traversal_tree(tree)
        sid = ctx.upload(warm.scene)
        ctx.render(sid, warm.settings)
    for method in ("sah", "lbvh"):
        ctx.build_bvh_device(warm.scene, method)
    big_frame(ctx, sid)
    held = fill(48 << 20)
    yield ctx, scene, nodes, sid, warm
    held.clear()
    torch.cuda.empty_cache()
    ctx.close()


@pytest.mark.parametrize("method", ["sah", "lbvh"])
def test_tree_build_takes_the_scratch(full, method):
    ctx, scene, nodes, sid, warm = full
    got, _ = ctx.build_bvh_device(scene, method)
    assert len(got) == 2 * scene.n_unified - 1
    if method == "lbvh":
        assert np.array_equal(got, nodes)
    ctx.render(sid, warm.settings)


@pytest.mark.parametrize("tree", [A.TRAVERSAL_UPLOADED, A.TRAVERSAL_LBVH, A.TRAVERSAL_SAH])
def test_upload_takes_the_scratch(full, tree):
    ctx, scene, nodes, sid, warm = full
    ctx.set_traversal_tree(tree)
    big = ctx.upload(scene, nodes)
    st = RenderSettings(width=64, height=48, samples=1, pathtrace=True, pathtrace_bounces=3,
                        block_size=128)
    a = ctx.render(big, st)
    ctx.free(big)
    assert np.isfinite(a).all()


def test_scenes_give_their_camera_nodes(gpu):
    """A scene that fits only where an earlier one's camera-relative nodes lie
    is accepted, and the earlier one renders the same image without them."""
    ctx = GpuContext(0)
    first, second = W.sphere_cloud(600_000).scene, W.sphere_cloud(150_000, seed=9).scene
    n1, _ = ctx.build_bvh_device(first, "lbvh")
    n2, _ = ctx.build_bvh_device(second, "lbvh")
    st = RenderSettings(width=96, height=64, samples=2, pathtrace=True, pathtrace_bounces=3,
                        block_size=128)
    sid = ctx.upload(second, n2)
    want2 = ctx.render(sid, st)
    ctx.free(sid)
    ctx.close()
    ctx = GpuContext(0)
    a = ctx.upload(first, n1)
    want1 = ctx.render(a, st)
    ctx.upload(W.sphere_cloud(100).scene)       # warm
    held = fill(8 << 20)
    b = ctx.upload(second, n2)
    held.clear()
    torch.cuda.empty_cache()
    assert np.array_equal(ctx.render(a, st), want1)
    assert np.array_equal(ctx.render(b, st), want2)
    ctx.close()


def test_adjoint_keeps_at_most_two_gigabytes(gpu):
    """The most records and bounces that the queued adjoint takes, in a frame
    of more paths than one chunk of them: the same gradients in chunks."""
    import dataclasses
    from conftest import load_golden
    from pencil_b200.scene import Light
    scene, _ = load_golden("three_spheres")
    scene.lights = [Light.point((k - 3.5, 4.0, -3.0), (0.1, 0.1, 0.1), 0.4) for k in range(8)]
    st = RenderSettings(width=1024, height=1030, samples=2, max_depth=16, pathtrace=True,
                        pathtrace_bounces=16, soft_shadow_samples=4)
    dl = np.random.default_rng(4).normal(size=(st.height, st.width, 3)).astype(np.float32)
    ctx = GpuContext(0)
    sid = ctx.upload(scene)
    nm, nl = scene.n_materials, len(scene.lights)
    b = ctx.adjoint(sid, dataclasses.replace(st, count_rays=True), dl, nm, nl, want_image=True)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    a = ctx.adjoint(sid, st, dl, nm, nl, want_image=True)
    torch.cuda.synchronize()
    taken = free - torch.cuda.mem_get_info()[0]
    assert 1 << 30 < taken <= (2 << 30) + (64 << 20)
    assert np.array_equal(a[3].view(np.uint32), b[3].view(np.uint32))
    for x, y in zip(a[:3], b[:3]):
        assert np.abs(x - y).max() <= 1e-9 * max(np.abs(y).max(), 1e-30)
    ctx.close()


@pytest.mark.parametrize("tree", [A.TRAVERSAL_UPLOADED, A.TRAVERSAL_LBVH])
def test_staging_grows_with_the_scenes(tree):
    """Uploads of one context whose staging is below 2 MB, above, below again
    (what is there is kept) and far above: each scene renders as it does in a
    context of its own."""
    ctx = GpuContext(0)
    ctx.set_traversal_tree(tree)
    for n in (300, 9_000, 300, 60_000, 9_000):
        w = W.sphere_cloud(n, 160, 90, 1, 3)
        own = GpuContext(0)
        own.set_traversal_tree(tree)
        a, b = (c.render(c.upload(w.scene), w.settings) for c in (ctx, own))
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), n
        own.close()
    ctx.close()
