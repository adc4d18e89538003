"""Batches without bounces (tile_kernel in batch.cu) against the oracle: tile shapes and
remainders, cameras in solid, empty, border and outside voxels, near and far world origins,
sun rays, iteration caps and the three traversal modes.  Every record word is equal, in the
12-byte form too."""
import copy

import numpy as np
import pytest

import voxelrt_gb300 as v
from tests.helpers import both_worlds, oracle_view

pytestmark = pytest.mark.gpu
SUN = np.array([0.3, 0.8, 0.5], np.float64) / np.linalg.norm([0.3, 0.8, 0.5])
SIZES = [(1, 1), (7, 5), (8, 8), (9, 17), (33, 31), (64, 64), (100, 3), (257, 40)]


def words(a):
    return np.ascontiguousarray(a).view(np.uint32).reshape(-1, 4)


def cameras(rng, edge, mode):
    """Eyes inside, on the clip box's sides, outside, and in a far frame (the same eye with its
    world origin moved 2^17 voxels away, so the ray origin is far from it)."""
    out = []
    for i, wh in enumerate(SIZES * 2):
        pos = rng.uniform(0, edge, 3)
        if i % 4 == 1:
            pos[i % 3] = [0.0, 1.0, edge - 1.0, edge][i // 4]
        elif i % 4 == 3:
            pos = pos * 3 - edge
        cam = v.look_at(pos, rng.uniform(0.2 * edge, 0.8 * edge, 3), 75.0, *wh)
        if i % 8 == 6:
            cam.world_origin[1] -= 1 << 17
            cam.origin[1] += 1 << 17
        out.append(v.make_view(cam, world=0, max_iters=[0, 1, 2, 64][i % 4], shadow_dir=SUN if i % 3 else None, **mode))
    return out


@pytest.fixture(scope="module")
def worlds(gpu):
    made = [both_worlds(v.synth_mix(96, seed=21)), both_worlds(v.synth_terrain((128, 64, 128), base=24, amplitude=20, seed=3))]
    yield made
    for w, _ in made:
        w.close()


@pytest.mark.parametrize("mode", [{}, dict(glsl=True), dict(aniso=True)], ids=["cpu", "glsl", "aniso"])
@pytest.mark.parametrize("cfg", [{}, dict(morton=1, tile_w=8, tile_h=8, chunk_tiles=3), dict(tile_w=16, tile_h=4),
                                 dict(tile_w=32, tile_h=1, chunk_tiles=7, warps_per_block=16), dict(warps_per_block=1,
                                                                                                    blocks_per_sm=1)])
def test_tiles_match_oracle(worlds, mode, cfg):
    rng = np.random.default_rng(7)
    views = cameras(rng, 96, mode)
    for vw in cameras(rng, 64, mode):
        vw = copy.copy(vw)
        vw.world = 1
        views.append(vw)
    want = [oracle_view(worlds[vw.world][1], vw) for vw in views]
    keys = ("tile_w", "tile_h", "morton", "warps_per_block", "blocks_per_sm", "refill_threshold", "chunk_tiles", "inner_iters")
    with_cfg = v.Batch([w for w, _ in worlds], views, v.BatchConfig(**{k: cfg.get(k, 0) for k in keys}))
    hits = with_cfg.run()
    for i in range(len(views)):
        assert np.array_equal(words(with_cfg.view_hits(hits, i)), words(want[i])), i
    # the kernel's own 12-byte records
    assert np.array_equal(with_cfg.run_packed().view(np.uint32), v.pack_hits(hits).view(np.uint32))
    assert with_cfg.stats()["rays_cast"] == sum(int((w["tag"] != v.NO_RAY).sum()) for w in want)
    with_cfg.close()


@pytest.mark.parametrize("n_views", [1, 2, 9])
def test_parts_deliver_every_record(worlds, n_views):
    """Batches of one, a few and several parts (vrt_batch_run cuts them by record count)."""
    rng = np.random.default_rng(n_views)
    views = [v.make_view(v.look_at(rng.uniform(0, 96, 3), rng.uniform(0, 96, 3), 70.0, 1280, 720), world=0,
                         shadow_dir=SUN if i % 2 else None) for i in range(n_views)]
    b = v.Batch([w for w, _ in worlds], views)
    hits = b.run()
    for i in range(n_views):
        assert np.array_equal(words(b.view_hits(hits, i)), words(oracle_view(worlds[0][1], views[i]))), i
    assert np.array_equal(b.run_packed().view(np.uint32), v.pack_hits(hits).view(np.uint32))
    b.close()
