"""The warp sums of the forward wall-normal pass on the host (CPU, no GPU):
each (parity, value) is stored by exactly one lane, and that lane holds its sum."""
import os
import subprocess

NATIVE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native")


def test_one_writer_per_value(tmp_path):
    exe = str(tmp_path / "paritysum_check")
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-I", "/usr/local/cuda/include", "-x", "c++",
                        os.path.join(NATIVE, "paritysum_check.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    rows = [[int(x) for x in ln.split()]
            for ln in subprocess.run([exe], capture_output=True, text=True, check=True).stdout.splitlines()]
    assert {6, 10} <= {nv for nv, _, _ in rows}
    for nv, not_one_writer, wrong in rows:
        assert not_one_writer == 0 and wrong == 0, (nv, not_one_writer, wrong)
