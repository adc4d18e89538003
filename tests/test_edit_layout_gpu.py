"""Sector layouts under edits (edit_sectors_kernel) against the oracle: batches around the 32
edits a warp tests at a time, sectors that gain and lose bricks in one batch, full sectors
packed in place around bricks no edit visits, and the group masks and table entries that
follow (casts in the three modes read them)."""
import numpy as np
import pytest

import voxelrt_gb300 as v
from tests.helpers import both_worlds, dense_to_stream
from tests.test_edit_gpu import assert_worlds_equal

pytestmark = pytest.mark.gpu


def stroke(rng, n, lo, hi, radius):
    e = np.zeros(n, v.EDIT_DTYPE)
    e["center"] = rng.integers(lo, hi, (n, 3))
    e["radius"] = rng.integers(0, radius + 1, n)
    kind = rng.integers(0, 3, n)
    e["material"] = np.where(kind == 0, 0, rng.integers(1, 256, n))
    e["mode"] = kind == 2
    return e


@pytest.mark.parametrize("n_edits", [1, 31, 32, 33, 70])
@pytest.mark.parametrize("fill", [0.0, 0.002, 1.0])
def test_layouts(gpu, n_edits, fill):
    """16x1x5 sectors: 8 sector groups, so a local stroke updates a list of them."""
    rng = np.random.default_rng(n_edits)
    vol = ((rng.random((32, 160, 512)) < fill) * rng.integers(1, 256, (32, 160, 512))).astype(np.uint8)
    w, o = both_worlds(dense_to_stream(vol) if fill else v.SectorData((16, 1, 5), [], [], np.zeros((0, 512), np.uint8)))
    rays = v.random_rays((512, 32, 160), seed=2, n=20_000)
    for step in range(4):
        lo = np.array([rng.integers(0, 440), -4, rng.integers(0, 100)])
        e = stroke(rng, n_edits, lo, lo + np.array([60, 40, 50]), 12)
        w.edit(e)
        o.edit(e)
        if step == 2:  # a whole sector carved around one corner brick, then part of it filled
            e = np.zeros(2, v.EDIT_DTYPE)
            e["center"], e["radius"], e["material"] = [(48, 16, 48), (33, 1, 33)], [20, 2], [0, 9]
            w.edit(e)
            o.edit(e)
        assert_worlds_equal(w, o)
        for mode in ({}, dict(glsl=True), dict(aniso=True)):
            want = o.cast(rays, glsl=bool(mode), aniso=mode.get("aniso", False))
            assert np.array_equal(w.cast(rays, **mode).view(np.uint32), want.view(np.uint32))
    w.close()
