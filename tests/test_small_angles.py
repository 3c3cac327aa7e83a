"""The sine of the block-floating-point sweeps (csrc/bfp.cuh, host instantiation) relative to itself."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(np.finfo(np.longdouble).nmant < 63, reason="no extended precision to compare with")
def test_relative_error_of_the_sine_down_to_small_angles(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "small_angle_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-w", "-I", os.path.join(HERE, "..", "sapien_gb300", "csrc"),
                    os.path.join(HERE, "small_angle_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    got = {w[0]: float(w[1]) for w in (line.split() for line in out.splitlines())}
    # the angle rounded to 2^-60 and the product cut off there, at an angle of 2^-16 and more
    assert got["relative"] <= 1.5 * 2.0**-44
    assert got["predicate"] == 1
