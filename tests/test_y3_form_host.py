"""Precision of getUVW in the backward wall-normal pass (CPU, no GPU): the
derivative sweeps are FP64 wherever the block form, which serves the same
lengths, was the only form; the mixed form has FP32 sweeps at six lengths."""
import os
import subprocess

NATIVE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native")
FP32_SWEEPS = {128, 192, 256, 384, 512, 768}


def test_sweep_precision(tmp_path):
    exe = str(tmp_path / "y3form_check")
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-I", "/usr/local/cuda/include", "-x", "c++",
                        os.path.join(NATIVE, "y3form_check.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    rows = [[int(x) for x in ln.split()]
            for ln in subprocess.run([exe], capture_output=True, text=True, check=True).stdout.splitlines()]
    assert FP32_SWEEPS < {m for m, _, _ in rows}
    for m, mixed, fp64 in rows:
        assert fp64 == 16
        assert mixed == (8 if m in FP32_SWEEPS else 16), m
