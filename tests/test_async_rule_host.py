"""Which kernel an asynchronous run takes is a rule on slots, sizes and the plan's regions, checked on the host: the
faster kernel runs only where its modularity was measured to be the other's (8 slots, large skewed graphs)."""
import os
import subprocess

from conftest import ROOT


def test_fast_kernel_only_where_measured(tmp_path):
    exe = str(tmp_path / "async_rule")
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    subprocess.run([cxx, "-std=c++17", "-O2", "-Wall", "-I", os.path.join(ROOT, "rak-lowmem-communities-cuda_b200", "csrc"),
                    "-I", os.path.join(ROOT, "include"), "-I", "/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "cpp", "async_rule.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
