"""The rules that pick a launch's kernel and claim size, on the host (no GPU): tests/cpp/
launch_rule_test.cpp links the product library and calls its planner at both sides of each
line."""
import subprocess

import pytest

from tests.test_plan_cpu import ROOT, build, cuda_include

SRC = ROOT / "tests" / "cpp" / "launch_rule_test.cpp"
EXE = ROOT / "tests" / "cpp" / "_build" / "launch_rule_test"


def test_kernel_and_claims():
    inc = cuda_include()
    if inc is None:
        pytest.skip("CUDA runtime headers not found")
    lib = build.build_library()
    EXE.parent.mkdir(exist_ok=True)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(ROOT / "include"), "-I", str(build.CSRC), "-I", str(inc),
                    str(SRC), "-L", str(lib.parent), "-lvrt", f"-Wl,-rpath,{lib.parent}", "-o", str(EXE)], check=True)
    res = subprocess.run([str(EXE)], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout + res.stderr
    assert "ok: 0 failures" in res.stdout
