"""CPU test of the integer-pipe double-precision arithmetic (csrc/sf_f64_int.cuh): every function bit for bit equal
to the host's own operation, on edge significands, zeros and seeded random values over the accepted range.  The device
code compiles the same functions."""
import os
import subprocess

from conftest import ROOT


def test_integer_double_arithmetic_matches_host():
    src = os.path.join(ROOT, "tests", "cpp", "f64_int_check.cpp")
    out_dir = os.path.join(ROOT, "oracle", "_build")
    os.makedirs(out_dir, exist_ok=True)
    exe = os.path.join(out_dir, "f64_int_check")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                           os.path.join(ROOT, "simferrofluid-cuda_gb300", "csrc"), src, "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True)
    bad, n = (int(v) for v in r.stdout.split()[-2:])
    assert r.returncode == 0 and bad == 0, r.stdout
    assert n > 20_000_000
