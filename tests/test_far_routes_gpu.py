"""The other ways to a far view's kernel (world origins beyond the fast step's, launch rules far_launch
and tile_launch), against the oracle: the entry point without allocations, the request server in
both modes, packed records, graph launches, and a batch whose cameras move between near and far
frames after its kernel was chosen.  Every record word is equal."""
import ctypes as C

import numpy as np
import pytest

import voxelrt_gb300 as v
from tests.helpers import both_worlds, oracle_view

pytestmark = pytest.mark.gpu
SUN = np.array([0.3, 0.8, 0.5], np.float64) / np.linalg.norm([0.3, 0.8, 0.5])
MODES = [{}, dict(glsl=True), dict(aniso=True)]
KINDS = [{}, dict(shadow_dir=SUN), dict(n_bounces=2), dict(n_bounces=2, shadow_dir=SUN)]
FRAMES = [(0, 0, 0), (1 << 22, 0, 0), (0, -(1 << 22) - 1, 3), (-(1 << 23), 1 << 23, 0)]


@pytest.fixture(scope="module")
def world(gpu):
    w, o = both_worlds(v.synth_terrain((128, 128, 128), base=54.0, amplitude=32.0, seed=3))
    yield w, o
    w.close()


def words(a):
    return np.ascontiguousarray(a).view(np.uint32).reshape(-1, 4)


def camera(i, frame):
    """Eyes in the open, one in the plane of an empty brick's face, in a frame moved by `frame`."""
    eye = np.array([(64.0, 100.0, 64.0), (40.3, 110.2, 70.7), (90.1, 96.5, 20.2)][i % 3])
    cam = v.look_at(eye, eye + (40 - 30 * i, -50, 35), 80.0, (47, 90, 33)[i % 3], (31, 17, 60)[i % 3])
    for c in range(3):
        cam.world_origin[c] += frame[c]
        cam.origin[c] -= frame[c]
    return cam


def views_of(kind, mode, frames=FRAMES):
    return [v.make_view(camera(i, f), **kind, **mode) for i, f in enumerate(frames)]


@pytest.mark.parametrize("mode", MODES, ids=lambda m: "+".join(m) or "cpu")
@pytest.mark.parametrize("kind", KINDS, ids=lambda k: "+".join(k) or "primary")
def test_static_and_batches(world, mode, kind):
    import torch
    w, o = world
    views = views_of(kind, mode)
    want = np.concatenate([words(oracle_view(o, vw)) for vw in views])
    out = torch.full((len(want), 4), -1, dtype=torch.int32, device="cuda")
    wh = (C.c_void_p * 1)(w.handle.value)
    v.capi.check(v.lib().vrt_render_views_static(wh, 1, (v.View * len(views))(*views), len(views), None, v.capi.ptr(out),
                                                 None))
    torch.cuda.synchronize()
    assert np.array_equal(words(out.cpu().numpy()), want)
    b = v.Batch([w], views)
    assert b.total_records == len(want)
    for graph in (True, True, False):
        out.fill_(-1)
        b.launch(out, graph=graph)
        torch.cuda.synchronize()
        assert np.array_equal(words(out.cpu().numpy()), want)
    assert np.array_equal(b.run_packed().view(np.uint32), v.pack_hits(want.view(v.HIT_DTYPE).reshape(-1)).view(np.uint32))
    b.close()


@pytest.mark.parametrize("mode", MODES, ids=lambda m: "+".join(m) or "cpu")
@pytest.mark.parametrize("kind", KINDS, ids=lambda k: "+".join(k) or "primary")
def test_cameras_that_move_between_frames(world, mode, kind):
    """The batch's kernel follows its first views; its records do not."""
    w, o = world
    near, far = [(0, 0, 0)] * 4, FRAMES[::-1]
    for start in (near, far):
        b = v.Batch([w], views_of(kind, mode, start))
        for frames in (far, near, far):
            views = views_of(kind, mode, frames)
            b.update_cameras([vw.cam for vw in views])
            hits = b.run()
            for i, vw in enumerate(views):
                assert np.array_equal(words(b.view_hits(hits, i)), words(oracle_view(o, vw))), (frames, i)
        b.close()


@pytest.mark.parametrize("resident", [True, False], ids=["resident", "launches"])
@pytest.mark.parametrize("mode", MODES, ids=lambda m: "+".join(m) or "cpu")
def test_server(world, mode, resident):
    w, o = world
    views = [vw for kind in KINDS for vw in views_of(kind, mode)]
    srv = v.Server([w], resident=resident)
    outs = [np.zeros(v.view_records(vw), v.HIT_DTYPE) for vw in views]
    for t in [srv.submit_render(vw, x) for vw, x in zip(views, outs)]:
        assert srv.wait(t)["status"] == 0
    srv.close()
    for vw, x in zip(views, outs):
        assert np.array_equal(words(x), words(oracle_view(o, vw)))
