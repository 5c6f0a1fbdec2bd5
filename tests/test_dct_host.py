"""The pruned DCT of the wall-normal passes on the host (CPU, no GPU): every
plan, one, three and six lines, whole and zero-padded inputs, against a
long-double DFT.  Tolerances as for the other FFT engines: FP64 2e-15, FP32
5e-7 of the largest output magnitude."""
import os
import subprocess

NATIVE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native")


def test_every_plan(tmp_path):
    exe = str(tmp_path / "ydct_check")
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-I", "/usr/local/cuda/include", "-x", "c++",
                        os.path.join(NATIVE, "ydct_check.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    rows = [ln.split() for ln in subprocess.run([exe], capture_output=True, text=True, check=True).stdout.splitlines()]
    assert len(rows) >= 38
    for prec, m, *errs in rows:
        assert all(float(e) < (2e-15 if prec == "double2" else 5e-7) for e in errs), (prec, m, errs)
