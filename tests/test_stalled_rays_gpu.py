"""Explicit rays that stand still until the iteration cap (stalled in trace_core.cuh) against the
oracle, which traces every step: caps around the slices and around rayCastCoarse's iteration 31,
and the ray counts of both cast kernels.  Every record word is equal."""
import numpy as np
import pytest

import voxelrt_gb300 as v
from tests.helpers import both_worlds

pytestmark = pytest.mark.gpu
MODES = [{}, dict(glsl=True), dict(aniso=True), dict(coarse=True), dict(aniso=True, coarse=True)]


@pytest.fixture(scope="module")
def world(gpu):
    w, o = both_worlds(v.synth_terrain((128, 128, 128), base=54.0, amplitude=32.0, seed=3))
    yield w, o
    w.close()


def make_rays(n):
    """Random rays, every third with one or two direction components of 0 or next to it."""
    rays = v.random_rays((128, 128, 128), seed=4, n=n)
    rng = np.random.default_rng(5)
    small = rng.choice(np.array([0.0, -0.0, 1e-7, -1e-5, 1e-3], np.float32), size=(n, 3))
    mask = rng.random((n, 3)) < 0.5
    mask[:, 0] &= ~(mask[:, 1] & mask[:, 2])
    mask[np.arange(n) % 3 != 0] = False
    rays["dir"] = np.where(mask, small, rays["dir"])
    return rays


def words(a):
    return np.ascontiguousarray(a).view(np.uint32)


@pytest.mark.parametrize("mode", MODES, ids=lambda m: "+".join(m) or "cpu")
@pytest.mark.parametrize("n", [3001, (1 << 18) + 37, (3 << 18) + 5])
def test_caps(world, mode, n):
    w, o = world
    rays = make_rays(n)
    caps = (0, 1, 7, 8, 9, 15, 16, 17, 30, 31, 32, 33, 39, 40, 41, 48, 96, 97, 200) if n < 10000 else (0, 30, 63)
    for cap in caps:
        got = w.cast(rays, max_iters=cap, **mode)
        want = o.cast(rays, max_iters=cap, **dict(mode, glsl=bool(mode)))  # the oracle's flag for all three
        assert np.array_equal(words(got), words(want)), cap
    # rays that reach the cap (rayCastCoarse has one of its own, and in CPU mode they are few)
    if not mode.get("coarse") and (mode or n > 10000):
        assert (got["steps"] == cap).any()  # rays that reach the cap
