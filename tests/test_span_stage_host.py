"""The tensor copies of the forward spanwise pass on the host (CPU, no GPU).

A tiled copy needs a 128-byte aligned destination and at most 256 rows; the
copies of a line cover it once and stay in the warp's part of shared memory,
whose first 128-byte boundary may lie up to 127 bytes in."""
import os
import subprocess

NATIVE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native")


def test_copy_destinations(tmp_path):
    exe = str(tmp_path / "zstage_check")
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-I", "/usr/local/cuda/include", "-x", "c++",
                        os.path.join(NATIVE, "zstage_check.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    rows = [[int(x) for x in ln.split()]
            for ln in subprocess.run([exe], capture_output=True, text=True, check=True).stdout.splitlines()]
    assert len(rows) == 22
    taken = {}
    for L, ok, part, *copies in rows:
        if not ok:
            continue
        copies = [copies[i:i + 3] for i in range(0, len(copies), 3)]
        taken[L] = len(copies)
        at = 0
        for first, n, offset in copies:
            assert first == at and 0 < n <= 256, (L, copies)
            assert offset % 128 == 0 and 128 + offset + n * 16 <= part, (L, copies, part)
            at += n
        assert at == L
    # the lengths that a whole copy serves, not multiples of 16 among them, and those of two halves
    assert all(taken.get(L) == 1 for L in (24, 36, 54, 72, 108, 144, 162, 192, 216, 256))
    assert all(taken.get(L) == 2 for L in (288, 384, 512))
