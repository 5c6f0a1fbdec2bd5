"""Which fields of one transform call share launches (CPU, no GPU).

The fields of a call go in order: a field whose output another one reads or
writes must not be in flight with it, whatever buffers a caller passes."""
import os
import subprocess

NATIVE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native")


def test_fields_that_share_memory(tmp_path):
    exe = str(tmp_path / "fields_check")
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-I", "/usr/local/cuda/include", "-x", "c++",
                        os.path.join(NATIVE, "fields_check.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([exe], capture_output=True, text=True, check=True).stdout.splitlines()
    rows = {ln.split()[0]: [int(x) for x in ln.split()[1:]] for ln in out}
    assert rows["random"][0] == 20000 and rows["random"][1] == 0  # no overlap goes unseen
    # (backward, forward): 1 = launches shared
    assert rows["apart"] == [1, 1]
    assert rows["same_points"] == [0, 1]  # forward only reads them
    assert rows["same_pencils"] == [0, 0]
    assert rows["in_place"] == [1, 1]  # each field on itself only
    assert rows["next_pencils"] == [0, 0]
    assert rows["interleaved"] == [1, 1]
