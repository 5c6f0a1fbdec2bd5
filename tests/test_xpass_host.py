"""The streamwise and the two-butterfly lines on the host (CPU, no GPU): every
plan of csrc/xpass.cuh and csrc/zpass.cuh in both precisions.

Transforms: FP64 2e-15, FP32 5e-7 of the largest output magnitude, as for the
other FFT engines.  Twiddles: rounded to nearest in both parts, so within half a
unit in the last place of a number below 1 in each, 2^-54 sqrt 2 (FP32 2^-25
sqrt 2, and one part in 1e6 for rounding by way of FP64)."""
import math
import os
import subprocess

NATIVE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native")


def test_every_plan(tmp_path):
    exe = str(tmp_path / "xpass_check")
    r = subprocess.run(["g++", "-O1", "-std=c++17", "-I", "/usr/local/cuda/include", "-x", "c++",
                        os.path.join(NATIVE, "xpass_check.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    rows = [ln.split() for ln in subprocess.run([exe], capture_output=True, text=True, check=True).stdout.splitlines()]
    assert len(rows) == 4 * 22
    for form, prec, length, tw, *errs in rows:
        fp64 = prec == "double2"
        assert float(tw) <= math.sqrt(2) * (2.0 ** -54 if fp64 else 2.0 ** -25 * (1 + 1e-6)) * (1 + 1e-3), (form, prec, length, tw)
        assert all(float(e) < (2e-15 if fp64 else 5e-7) for e in errs), (form, prec, length, errs)
