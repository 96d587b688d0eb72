"""CPU test of the integer seven-point sum of the mixed form's FP64 residual (csrc/sf_f64_int.cuh, fixed_stencil): its error
against the exact sum, relative to the values of the sum itself, is within its stated bound and no larger than that of FP64
arithmetic.  The device compiles the same function."""
import os
import subprocess

from conftest import PKG_NAME, ROOT


def test_integer_stencil_loses_no_more_than_fp64():
    out_dir = os.path.join(ROOT, "oracle", "_build")
    os.makedirs(out_dir, exist_ok=True)
    exe = os.path.join(out_dir, "fixed_stencil_check")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, PKG_NAME, "csrc"),
                           os.path.join(ROOT, "tests", "cpp", "fixed_stencil_check.cpp"), "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True)
    bad, n = (int(v) for v in r.stdout.split()[-2:])
    assert r.returncode == 0 and bad == 0, r.stdout
    assert n > 6_000_000
