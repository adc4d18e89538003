"""The ray chunks of the persistent cast kernel (cast_queue.h) on the host, no GPU: no ray in no
chunk or in two, up to 2^32 - 1 rays."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
SRC = ROOT / "tests" / "cpp" / "cast_queue_test.cpp"
EXE = ROOT / "tests" / "cpp" / "_build" / "cast_queue_test"


def test_every_ray_lies_in_one_chunk():
    EXE.parent.mkdir(exist_ok=True)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(ROOT / "include"), "-I", str(ROOT / "voxelrt_gb300" / "csrc"),
                    str(SRC), "-o", str(EXE)], check=True)
    res = subprocess.run([str(EXE)], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout + res.stderr
    assert "ok: 0 failures" in res.stdout
