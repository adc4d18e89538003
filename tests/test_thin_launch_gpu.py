"""Small launches (thin_lanes_log2 in thin_launch.cuh: 4 to 32 rays per warp) against the oracle, at
the ray counts where the rays per warp change and at the remainders of a warp and a block;
frames, paths and G-buffers of odd shapes likewise.  Every record word is equal."""
import numpy as np
import pytest

import voxelrt_gb300 as v
from tests.helpers import both_worlds, oracle_view

pytestmark = pytest.mark.gpu
# n >> (l - 1) <= 2432 warps (4 rays a warp up to 9728 rays, 8 to 19456, 16 to 38912)
COUNTS = [1, 3, 4, 5, 31, 33, 127, 2000, 9728, 9731, 19456, 19459, 38911, 38915]
SHAPES = [(1, 1), (3, 2), (64, 64), (76, 64), (77, 64), (4864, 1), (1, 4866), (139, 70), (128, 76), (195, 100), (140, 139), (256, 152),
          (195, 200)]


@pytest.fixture(scope="module")
def world(gpu):
    w, o = both_worlds(v.synth_mix(96, seed=5))
    yield w, o
    w.close()


def words(a):
    return np.ascontiguousarray(a).view(np.uint32)


@pytest.mark.parametrize("mode", [{}, dict(glsl=True), dict(coarse=True), dict(aniso=True)], ids=lambda m: "+".join(m) or "cpu")
def test_casts(world, mode):
    w, o = world
    rays = v.random_rays((96, 96, 96), seed=9, n=max(COUNTS))
    want = words(o.cast(rays, glsl=bool(mode), coarse=mode.get("coarse", False), aniso=mode.get("aniso", False)))
    for n in COUNTS:
        assert np.array_equal(words(w.cast(rays[:n], **mode)), want[: 4 * n]), n


@pytest.mark.parametrize("shape", SHAPES)
def test_frames(world, shape):
    w, o = world
    for pos in ((50.3, 70.1, 20.7), (-30.0, 60.0, 48.0)):  # inside, outside the world
        cam = v.look_at(pos, (48, 40, 48), 70.0, *shape)
        assert np.array_equal(words(w.render_view(cam)), words(o.render_view(cam)))


@pytest.mark.parametrize("mode", [{}, dict(glsl=True), dict(aniso=True)], ids=lambda m: "+".join(m) or "cpu")
def test_paths_and_gbuffers(world, mode):
    w, o = world
    palette, proj = np.arange(256, dtype=np.uint32), np.eye(4, dtype=np.float32).reshape(16)
    for i, shape in enumerate(SHAPES):
        cam = v.look_at((50.3, 70.1, 20.7), (48, 40, 48), 70.0, *shape)
        view = v.make_view(cam, n_bounces=i % 3, shadow_dir=(0.35, 0.8, 0.48) if i % 2 else None, **mode)
        assert np.array_equal(words(v.render_path(w, view)), words(oracle_view(o, view))), shape
        tex, depth = v.render_gbuffer(w, v.make_view(cam, **mode), palette, proj)
        want_tex, want_depth, _ = o.render_gbuffer(cam, palette, proj, **mode)
        assert np.array_equal(tex, want_tex) and np.array_equal(words(depth), words(want_depth)), shape
