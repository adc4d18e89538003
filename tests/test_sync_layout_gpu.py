"""Sync batches (sync_sectors_kernel) against the oracle: full sectors and single bricks, kept
bricks that move, fresh bricks without bytes, deleted sectors, sectors outside the world, the
same sector twice in one call, and more sectors than the first pinned list holds."""
import numpy as np
import pytest

import voxelrt_gb300 as v
from tests.helpers import both_worlds
from tests.test_edit_gpu import assert_worlds_equal

pytestmark = pytest.mark.gpu


def mask_of(rng, share):
    return int(sum(1 << b for b in range(64) if rng.random() < share))


@pytest.mark.parametrize("extent,n", [((2, 1, 2), 5), ((4, 3, 5), 70), ((16, 8, 16), 1900)])
def test_sync_batches(gpu, extent, n):
    rng = np.random.default_rng(n)
    w, o = both_worlds(v.SectorData(extent, [], [], np.zeros((0, 512), np.uint8)))
    brick = (rng.random((64, 512)) < 0.05) * rng.integers(1, 256, (64, 512))
    brick[7] = 0
    masks = {}
    for step in range(4):
        idx, alloc, dirty, bricks = [], [], [], []
        for i in range(n):
            c = [int(rng.integers(-1 if step == 3 else 0, e)) for e in extent]  # (some outside in the last call)
            s = v.sector_index(*c)
            old = masks.get(s, 0)
            a = [0, (1 << 64) - 1, 1 << int(rng.integers(64)), old | mask_of(rng, 0.1), old & mask_of(rng, 0.7),
                 mask_of(rng, 0.5)][int(rng.integers(6))]
            # supplied bricks: all new ones, or (from the second call on) some left to zeros and the old content
            d = a & (mask_of(rng, 0.5) if step else (1 << 64) - 1)
            idx.append(s), alloc.append(a), dirty.append(d)
            bricks += [brick[int(k)] for k in rng.integers(0, 64, bin(d).count("1"))]
            if all(0 <= x < e for x, e in zip(c, extent)):
                masks[s] = a
        b = np.array(bricks, np.uint8).reshape(-1, 512)
        args = (np.array(idx, np.int32), np.array(alloc, np.uint64), b, np.array(dirty, np.uint64))
        w.sync_sectors(*args)
        o.sync_sectors(*args)
        assert_worlds_equal(w, o)
        rays = v.random_rays([32 * e for e in extent], seed=step, n=5_000)
        for mode in ({}, dict(glsl=True), dict(aniso=True)):
            want = o.cast(rays, glsl=bool(mode), aniso=mode.get("aniso", False))
            assert np.array_equal(w.cast(rays, **mode).view(np.uint32), want.view(np.uint32))
    w.close()
