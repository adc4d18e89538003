"""Which bricks an edit's sphere reaches (edit_geometry.h) on the host, no GPU: the test of a whole
sector at once against that of each of its bricks."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
SRC = ROOT / "tests" / "cpp" / "edit_geometry_test.cpp"
EXE = ROOT / "tests" / "cpp" / "_build" / "edit_geometry_test"


def test_sector_at_once_equals_every_brick():
    EXE.parent.mkdir(exist_ok=True)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(ROOT / "include"), "-I", str(ROOT / "voxelrt_gb300" / "csrc"),
                    str(SRC), "-o", str(EXE)], check=True)
    res = subprocess.run([str(EXE)], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout + res.stderr
    assert "ok: 0 failures" in res.stdout
