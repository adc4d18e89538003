"""Sectors listed several times in a call and over several calls (the batch numbers by which
vrt_world_sync_sectors knows the sectors of its present batch): each later record follows the
earlier, as in the oracle's world."""
import numpy as np
import pytest

import voxelrt_gb300 as v
from oracle.oracle import OracleWorld

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sectors", [(2, 1, 2), (64, 32, 64)])
def test_repeated_sectors(gpu, sectors):
    rng = np.random.default_rng(sectors[0])
    w, o = v.World(sectors), OracleWorld(sectors)
    names = [(0, 0, 0), (1, 0, 1), (sectors[0] - 1, sectors[1] - 1, sectors[2] - 1)]
    state = {}
    for call in range(6):
        pick = [names[int(k)] for k in rng.integers(0, len(names), (1, 4, 9)[call % 3])]
        idx, masks, dirty, bricks = [], [], [], []
        for s in pick:
            m = int(rng.integers(0, 1 << 62)) & int(rng.integers(0, 1 << 62))
            old, data = state.get(s, (0, {}))
            d = m & (~old | int(rng.integers(0, 1 << 62)))  # new bricks have bytes, of the others some
            data = {b: x for b, x in data.items() if m >> b & 1}
            for b in range(64):
                if d >> b & 1:
                    data[b] = rng.integers(0, 5, 512).astype(np.uint8)
                    bricks.append(data[b])
            state[s] = (m, data)
            idx.append(v.sector_index(*s)), masks.append(m), dirty.append(d)
        w.sync_sectors(idx, np.array(masks, np.uint64), np.array(bricks, np.uint8).reshape(-1, 512), np.array(dirty, np.uint64))
        for s, (m, data) in state.items():
            got, b = w.read_sector(v.sector_index(*s))
            assert got == m
            assert np.array_equal(b, np.array([data[k] for k in sorted(data)], np.uint8).reshape(-1, 512))
    idx = np.array([v.sector_index(*s) for s in state], np.int32)
    masks = np.array([m for m, _ in state.values()], np.uint64)
    o.upload(v.SectorData(sectors, idx, masks, np.array([d[k] for _, d in state.values() for k in sorted(d)], np.uint8)))
    rays = v.random_rays((64, 32, 64), seed=2, n=5_000)
    assert np.array_equal(w.cast(rays).view(np.uint32), o.cast(rays).view(np.uint32))
    w.close()
