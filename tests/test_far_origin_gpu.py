"""World origins far from the world, and ray origins as far from theirs, against the oracle: on
either side of the bounds that decide between the fast and the general step (trace_core.cuh:
kNearWorldOrigin, kFastOrigin, kFastInvDir), where most rays stand still until the iteration cap;
explicit rays, views, G-buffers and batches on the GPU's own step, whose packed adds the host
build of the step does not have.  Every record word is equal."""
import numpy as np
import pytest

import voxelrt_gb300 as v
from tests.helpers import both_worlds, dense_to_stream, oracle_view
from tests.test_step_range_cpu import edge_rays

pytestmark = pytest.mark.gpu
SUN = np.array([0.3, 0.8, 0.5], np.float64) / np.linalg.norm([0.3, 0.8, 0.5])
MODES = [{}, dict(glsl=True), dict(aniso=True)]
FAR = [(0, 0, 0), (65537, -65537, 3), ((1 << 21) - 1, 5, -(1 << 21)), ((1 << 21) + 1, 0, 0), (0, -(1 << 21) - 1, 7),
       ((1 << 22) - 1, -(1 << 22), 1), (1 << 22, 0, -(1 << 22) - 1), (1 << 24, -(1 << 23), 0), (1 << 30, 0, -(1 << 30))]


def words(a):
    return np.ascontiguousarray(a).view(np.uint32)


@pytest.fixture(scope="module")
def world(gpu):
    rng = np.random.default_rng(8)
    vol = ((rng.random((64, 64, 96)) < 0.01) * rng.integers(1, 256, (64, 64, 96))).astype(np.uint8)
    vol[:4] = 9           # a floor, and walls on the grid's sides
    vol[:, :, 0] = 8
    vol[:, 63, 40:] = 7
    w, o = both_worlds(dense_to_stream(vol))
    yield w, o
    w.close()


@pytest.mark.parametrize("mode", MODES + [dict(coarse=True)], ids=lambda m: "+".join(m) or "cpu")
@pytest.mark.parametrize("wo", FAR)
def test_casts(world, mode, wo):
    w, o = world
    want = dict(mode, glsl=bool(mode))
    rays = edge_rays(np.random.default_rng(abs(sum(wo)) + len(mode)), (96, 64, 64), wo, 9_000)
    for n in (9_000, 1):
        got = w.cast(rays[:n], world_origin=wo, max_iters=200, **mode)
        assert np.array_equal(words(got), words(o.cast(rays[:n], world_origin=wo, max_iters=200, **want)))


@pytest.mark.parametrize("mode", MODES + [dict(coarse=True)], ids=lambda m: "+".join(m) or "cpu")
@pytest.mark.parametrize("wo", [(5, 0, -3), ((1 << 22) + 5, -(1 << 22), 1 << 23)])
def test_many_rays(world, mode, wo):
    """The persistent kernel's counts, near and far rays side by side in every warp."""
    w, o = world
    n = (3 << 18) + 77
    rays = np.resize(edge_rays(np.random.default_rng(4), (96, 64, 64), wo, 4_099), n)
    rays["tag"] = np.arange(n)
    want = np.resize(o.cast(rays[:4_099], world_origin=wo, max_iters=64, **dict(mode, glsl=bool(mode))), n)
    want["tag"] = rays["tag"]
    assert np.array_equal(words(w.cast(rays, world_origin=wo, max_iters=64, **mode)), words(want))


def view_of(wo, wh, i, mode, **kw):
    """A view of the world whose frame lies `wo` voxels off (the eye as near as floats allow)."""
    cam = v.look_at((48.3, 40.2, 30.7), (60.0 - 9 * i, 5.0 + 7 * i, 40.0), 80.0, *wh)
    for c in range(3):
        cam.world_origin[c] += wo[c]
        cam.origin[c] -= wo[c]
    return v.make_view(cam, max_iters=[0, 37][i % 2], **mode, **kw)


@pytest.mark.parametrize("mode", MODES, ids=lambda m: "+".join(m) or "cpu")
def test_views_and_batches(world, mode):
    w, o = world
    kinds = [{}, dict(shadow_dir=SUN), dict(n_bounces=2), dict(n_bounces=2, shadow_dir=SUN)]
    views, far = [], [wo for wo in FAR if max(map(abs, wo)) < 1 << 30]
    for i, wo in enumerate(far):
        for kw in kinds:
            views.append(view_of(wo, ((40, 23), (61, 33))[i % 2], i, mode, **kw))
    want = [oracle_view(o, vw) for vw in views]
    for vw, x in zip(views, want):
        assert np.array_equal(words(v.render_path(w, vw)), words(x)), vw.cam.world_origin[:]
    for first in range(4):  # primary rays, sun rays, bounces, whole paths: the far views among near ones
        some = list(range(first, len(views), 4))
        b = v.Batch([w], [views[i] for i in some])
        hits = b.run()
        for k, i in enumerate(some):
            assert np.array_equal(words(b.view_hits(hits, k)), words(want[i])), views[i].cam.world_origin[:]
        b.close()


@pytest.mark.parametrize("mode", MODES, ids=lambda m: "+".join(m) or "cpu")
def test_frames_and_gbuffers(world, mode):
    w, o = world
    palette, proj = np.arange(256, dtype=np.uint32), np.eye(4, dtype=np.float32).reshape(16)
    for i, wo in enumerate(FAR[:-1]):
        vw = view_of(wo, (57, 31), i, mode)
        if not mode:
            assert np.array_equal(words(w.render_view(vw.cam)), words(o.render_view(vw.cam)))
        tex, depth = v.render_gbuffer(w, v.make_view(vw.cam, **mode), palette, proj)
        want_tex, want_depth, _ = o.render_gbuffer(vw.cam, palette, proj, **mode)
        assert np.array_equal(tex, want_tex) and np.array_equal(words(depth), words(want_depth)), wo
