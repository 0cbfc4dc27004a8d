"""The compiled code does not depend on the machine that builds it: no split compilation, which divides a unit by the
number of processors (one unit came out as two different programs with 2 or 8 and with 4 or 16 of them, 2% apart in
speed), and the same flags for every CUDA unit."""
import os
import re
import subprocess

from conftest import PKG


def test_every_cuda_unit_has_the_same_flags():
    out = subprocess.run(["make", "-n", "-B", "-C", PKG], capture_output=True, text=True, check=True, timeout=60).stdout
    lines = [x for x in out.splitlines() if "-c " in x and ".cu " in x]
    assert len(lines) == len([f for f in os.listdir(os.path.join(PKG, "csrc")) if f.endswith(".cu")])
    assert "split-compile" not in out
    assert len({re.sub(r"-c \S+ -o \S+", "", x).strip() for x in lines}) == 1
