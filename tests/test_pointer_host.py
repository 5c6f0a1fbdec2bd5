"""Which device pointers of a caller a kernel takes directly (CPU, no GPU): the
context's own device's or managed memory, 16-byte aligned; another device's,
the host's and misaligned pencils go through copies."""
import os
import subprocess

NATIVE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native")


def test_direct_pointers(tmp_path):
    exe = str(tmp_path / "pointer_check")
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-I", "/usr/local/cuda/include", "-x", "c++",
                        os.path.join(NATIVE, "pointer_check.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    rows = [[int(x) for x in ln.split()]
            for ln in subprocess.run([exe], capture_output=True, text=True, check=True).stdout.splitlines()]
    assert len(rows) == 8
    for owner, dev, off, device, managed, host, unregistered in rows:
        assert device == (owner == dev and off == 0), (owner, dev, off)
        assert managed == (off == 0) and not host and not unregistered
