"""Batches whose claims are parts of a tile (launch_persistent in batch.cu): launches of one
64-ray tile a chunk, at the tile counts where the parts change (4 rays up to 152 tiles, 8 to
304, 16 to 608, 32 to 7,296; with bounces 32 from there on), with tiles that hang over the
view's edges, against the oracle.  Every record word is equal."""
import numpy as np
import pytest

import voxelrt_gb300 as v
from tests.helpers import both_worlds, oracle_view

pytestmark = pytest.mark.gpu
# tiles: shapes of the views
VIEWS = {1: [(3, 2)], 152: [(150, 63)], 153: [(72, 136)], 304: [(302, 64)], 305: [(488, 37)], 608: [(250, 150)],
         609: [(168, 232)], 7296: [(605, 768)], 7297: [(605, 768), (3, 2)]}
SUN = (0.35, 0.8, 0.48)


def words(a):
    return np.ascontiguousarray(a).view(np.uint32)


@pytest.fixture(scope="module")
def world(gpu):
    w, o = both_worlds(v.synth_mix(64, seed=8))
    yield w, o
    w.close()


def check(world, shapes, cfg, **kw):
    w, o = world
    views = [v.make_view(v.look_at((-20.0, 50.0, 30.5), (32, 20, 32), 70.0, *s), **kw) for s in shapes]
    want = np.concatenate([oracle_view(o, vw).reshape(-1) for vw in views])
    b = v.Batch([w], views, v.BatchConfig(chunk_tiles=1, **cfg))
    assert np.array_equal(words(b.run()), words(want)), (shapes, cfg, kw)
    assert np.array_equal(b.run_packed().view(np.uint32), v.pack_hits(want).view(np.uint32))
    b.close()


@pytest.mark.parametrize("tiles", VIEWS)
def test_tile_counts(world, tiles):
    assert sum(-(-w // 8) * -(-h // 8) for w, h in VIEWS[tiles]) == tiles
    check(world, VIEWS[tiles], {})
    check(world, VIEWS[tiles], {}, n_bounces=1)


@pytest.mark.parametrize("cfg", [dict(tile_w=8, tile_h=8, morton=1), dict(tile_w=16, tile_h=4), dict(tile_w=32, tile_h=1)],
                         ids=str)
@pytest.mark.parametrize("mode", [{}, dict(glsl=True), dict(aniso=True)], ids=lambda m: "+".join(m) or "cpu")
def test_tile_shapes(world, cfg, mode):
    for shape in ((33, 9), (150, 63), (301, 77), (500, 150)):
        check(world, [shape], cfg, shadow_dir=SUN, **mode)
        check(world, [shape], cfg, n_bounces=2, shadow_dir=SUN, **mode)
