"""Block-floating-point operations (csrc/bfp.cuh, host instantiation) are at least as exact as the
FP64 operations they stand for, against long double (64-bit mantissas or more)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(np.finfo(np.longdouble).nmant < 63, reason="no extended precision to compare with")
def test_operations_are_no_less_exact_than_fp64(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "bfp_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-w", "-I", os.path.join(HERE, "..", "sapien_gb300", "csrc"),
                    os.path.join(HERE, "bfp_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    got = {w[0]: [float(x) for x in w[1:]] for w in (line.split() for line in out.splitlines())}
    for name in ("cross", "rotate", "add", "scale"):
        assert got[name][0] <= got[name][1], (name, got[name])
    for name in ("sin", "cos", "reciprocal", "rsqrt"):  # below a rounding of FP64 near 1
        assert got[name][0] <= 2.0**-53, (name, got[name])
    assert got["rounding"][0] <= 2.0**-53 * (1 + 1e-9)  # results are rounded once, to nearest
    # halves at the ends of their range: two products, each off by the low product (2^-58 of the
    # norms' 2^120) and a rounding (2^-57); a negated mantissa by one unit
    assert got["edges"][0] <= 2.0**-55
