"""Unit-weight sketches of one-lane vertices keep whole numbers as the bits of (denormal) floats: the choice and the
move must not depend on whether the build flushes denormals."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.gpu
@pytest.mark.parametrize("flag", ["-ftz=false", "-ftz=true", "--use_fast_math"])
def test_choice_and_move_with_any_flags(tmp_path, flag):
    exe = tmp_path / "unit_order"
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    subprocess.run(["nvcc", "-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", "-ccbin", cxx, flag,
                    "-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "rak-lowmem-communities-cuda_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "unit_order.cu"), "-o", str(exe)], check=True, timeout=280)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
