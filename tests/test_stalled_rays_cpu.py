"""Rays that stand still (stalled in trace_core.cuh) on the host build of the device step, against
the oracle, which traces every step: rays on either side of every bound of the fast step, in all
modes, with caps around the slices and around rayCastCoarse's iteration 31.  Every record word is
equal, and in the far frames rays do end in hits and at the cap."""
import subprocess

import numpy as np
import pytest

import voxelrt_gb300 as v
from tests.helpers import dense_to_stream
from tests.test_device_logic_cpu import ROOT, oracle_for, run
from tests.test_step_range_cpu import MODES, edge_rays

EXE = ROOT / "tests" / "cpp" / "_build" / "stalled_test"


@pytest.fixture(scope="module")
def exe():
    EXE.parent.mkdir(exist_ok=True)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fno-fast-math", "-I", str(ROOT / "include"),
                    str(ROOT / "tests" / "cpp" / "stalled_test.cpp"), "-o", str(EXE)], check=True)
    return EXE


def world():
    rng = np.random.default_rng(8)
    vol = ((rng.random((64, 32, 96)) < 0.01) * rng.integers(1, 256, (64, 32, 96))).astype(np.uint8)
    vol[:4] = 9           # a floor, and walls on the grid's sides
    vol[:, :, 0] = 8
    vol[:, 31, 40:] = 7
    return dense_to_stream(vol)


@pytest.mark.parametrize("mode", MODES, ids=lambda m: "+".join(m) or "cpu")
@pytest.mark.parametrize("wo", [(0, 0, 0), (65536, -65537, 3), (1 << 21, -(1 << 21) - 1, 7), ((1 << 21) + 1, 0, 0),
                                ((1 << 22) - 1, -(1 << 22), 0), (1 << 22, 0, -(1 << 22) - 1), (1 << 24, 0, -(1 << 23)),
                                (1 << 30, -(1 << 30), 0)])
def test_records_equal_the_full_traversal(exe, tmp_path, mode, wo):
    data = world()
    rays = edge_rays(np.random.default_rng(abs(sum(wo)) + 3 * len(mode)), (96, 64, 32), wo, 8_000)
    oracle = oracle_for(data)
    for cap in (96,) if mode.get("coarse") else (200, 16, 33):
        got = run(exe, tmp_path, data, rays, cap, wo, **mode)
        want = oracle.cast(rays, world_origin=wo, max_iters=cap, **mode)
        bad = np.nonzero(got.view(np.uint32).reshape(-1, 4) != want.view(np.uint32).reshape(-1, 4))[0]
        assert bad.size == 0, (cap, len(np.unique(bad)), rays[bad[0]], got[bad[0]], want[bad[0]])
    hit = want["voxel"] != v.MISS_VOXEL
    if max(map(abs, wo)) <= 1 << 22:
        assert (hit & (want["steps"] > 0)).any()  # not only rays that start in solid voxels
    if 1 << 20 < max(map(abs, wo)) <= 1 << 24 and not mode.get("coarse"):
        assert (want["steps"] == cap).any()       # rays at the cap
