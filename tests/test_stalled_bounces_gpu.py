"""Rays that stand still in GLSL launches with bounces (kStall in batch.cu: the test between the slices
of the persistent kernel) against the oracle: cameras with coordinates on the face of an empty
brick, from which a third of the rays do, and others; slice lengths, refills and caps around them, and rayCastCoarse's
iteration 31.  Every record word is equal, and the counting launch traces every ray."""
import numpy as np
import pytest

import voxelrt_gb300 as v
from tests.helpers import both_worlds, oracle_view

pytestmark = pytest.mark.gpu
SUN = np.array([0.3, 0.8, 0.5], np.float64) / np.linalg.norm([0.3, 0.8, 0.5])


@pytest.fixture(scope="module")
def world(gpu):
    w, o = both_worlds(v.synth_terrain((128, 128, 128), base=54.0, amplitude=32.0, seed=3))
    yield w, o
    w.close()


def words(a):
    return np.ascontiguousarray(a).view(np.uint32).reshape(-1, 4)


@pytest.mark.parametrize("mode", [dict(glsl=True), dict(aniso=True)], ids=lambda m: "+".join(m))
@pytest.mark.parametrize("inner,refill", [(0, 0), (1, 32), (3, 28), (16, 1), (64, 20)])
def test_batches(world, mode, inner, refill):
    w, o = world
    views = []
    for i, cap in enumerate((0, 1, 30, 33, 48, 96, 200)):
        eye = np.array((64.0, 100.0, 64.0) if i % 2 else (60.3, 100.2, 50.7))
        cam = v.look_at(eye, eye + (-74 + 20 * i, -40, 44), 80.0, 70 + i, 41)
        views += [v.make_view(cam, n_bounces=3, max_iters=cap, **mode),
                  v.make_view(cam, n_bounces=2, max_iters=cap, shadow_dir=SUN, **mode)]
    want = [oracle_view(o, vw) for vw in views]
    assert (want[-4][0]["steps"] == 96).mean() > 0.1  # primary rays at the cap
    cfg = v.BatchConfig(0, 0, 0, 0, 0, refill, 0, inner)
    for kind in (0, 1):
        b = v.Batch([w], views[kind::2], cfg)
        hits = b.run()
        for k, x in enumerate(want[kind::2]):
            assert np.array_equal(words(b.view_hits(hits, k)), words(x)), k
        b.close()


@pytest.mark.parametrize("mode", [dict(glsl=True), dict(aniso=True)], ids=lambda m: "+".join(m))
def test_counts(world, mode):
    """Records and rays of the counting launch, which does not end stalled rays early."""
    import torch
    w, o = world
    views = [v.make_view(v.look_at((64.0, 100.0, 64.0), (40, 40, 90), 80.0, 96, 64), n_bounces=4, **mode)]
    b = v.Batch([w], views)
    out = torch.zeros((b.total_records, 4), dtype=torch.int32, device="cuda")
    stats = b.measure(out)
    want = oracle_view(o, views[0])
    cast = want["tag"] != v.NO_RAY
    assert np.array_equal(words(out.cpu().numpy()), words(want))
    assert stats["rays_cast"] == int(cast.sum())
    b.close()
