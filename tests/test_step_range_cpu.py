"""The fast step's bounds (trace_core.cuh: RayState::fast) against the oracle, on the host
build of the device step: rays whose origins, directions and world origins lie on either
side of every bound that decides between the fast and the general step.  Records are
bit formats, so they are equal word by word."""
import numpy as np
import pytest

import voxelrt_gb300 as v
from tests.helpers import dense_to_stream, make_rays
from tests.test_device_logic_cpu import exe, oracle_for, run  # noqa: F401 (exe is a fixture)

MODES = [dict(), dict(glsl=True), dict(glsl=True, coarse=True), dict(glsl=True, aniso=True)]


def edge_rays(rng, size, wo, n):
    """Origins at the clip box's and the grid's sides, a float beside them, inside, outside and
    far away; directions with zero, denormal, tiny and huge components."""
    size = np.array(size, np.float64)
    kind = rng.integers(0, 6, (n, 3))
    side = np.where(rng.random((n, 3)) < 0.5, 0.0, size)
    inner = np.where(side == 0, 1.0, size - 1.0)
    pos = np.choose(kind, [rng.uniform(0, size, (n, 3)), side, inner, np.floor(rng.uniform(0, size, (n, 3))),
                           side + rng.uniform(-40, 40, (n, 3)), rng.uniform(1, size - 1, (n, 3))])
    far = rng.random(n) < 0.05
    pos[far] = pos[far] * 10.0 ** rng.uniform(2, 9, (far.sum(), 1))
    o = (pos - np.array(wo, np.float64)).astype(np.float32)
    ulp = rng.integers(-1, 2, (n, 3))
    o = np.where(ulp < 0, np.nextafter(o, np.float32(-np.inf)), np.where(ulp > 0, np.nextafter(o, np.float32(np.inf)), o))
    d = rng.normal(size=(n, 3))
    scale = rng.choice([0.0, -0.0, 1e-42, 1e-30, 3e-29, 1e-6, 1e20], (n, 3))
    odd = rng.random((n, 3)) < 0.15
    return make_rays(o, np.where(odd, d * scale, d).astype(np.float32))


@pytest.mark.parametrize("mode", MODES, ids=lambda m: "+".join(m) or "cpu")
@pytest.mark.parametrize("wo", [(0, 0, 0), (37, -5, 60), (65536, -65536, 65535), (65537, 0, 0), (0, -65537, 3), (1 << 21, -(1 << 21), 7), ((1 << 21) + 1, 0, 0),
                                (1 << 22, 0, -(1 << 24)), (1 << 30, -(1 << 30), 0)])
def test_range_edges(exe, tmp_path, mode, wo):  # noqa: F811
    rng = np.random.default_rng(abs(sum(wo)) + len(mode))
    vol = ((rng.random((64, 32, 96)) < 0.01) * rng.integers(1, 256, (64, 32, 96))).astype(np.uint8)
    vol[:4] = 9           # a floor, and walls on the grid's sides: hits in the outermost voxels
    vol[:, :, 0] = 8
    vol[:, 31, 40:] = 7
    data = dense_to_stream(vol)
    rays = edge_rays(rng, (96, 64, 32), wo, 12_000)
    iters = 96 if mode.get("coarse") else 200
    got = run(exe, tmp_path, data, rays, iters, wo, **mode)
    want = oracle_for(data).cast(rays, world_origin=wo, max_iters=iters, **mode)
    bad = np.nonzero(got.view(np.uint32).reshape(-1, 4) != want.view(np.uint32).reshape(-1, 4))[0]
    assert bad.size == 0, (len(np.unique(bad)), rays[bad[0]], got[bad[0]], want[bad[0]])
    assert (want["voxel"] != v.MISS_VOXEL).any() or max(abs(c) for c in wo) > 1 << 16


def test_iteration_caps(exe, tmp_path):  # noqa: F811
    """Caps at, before and after the step that ends the ray."""
    rng = np.random.default_rng(5)
    vol = np.zeros((32, 32, 64), np.uint8)
    vol[::8, ::8, ::8] = 3
    data = dense_to_stream(vol)
    rays = edge_rays(rng, (64, 32, 32), (0, 0, 0), 3_000)
    for cap in (1, 2, 3, 5, 9):
        got, want = run(exe, tmp_path, data, rays, cap), oracle_for(data).cast(rays, max_iters=cap)
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), cap
