"""The bench's clock sampler (CPU, a stand-in for nvidia-smi): a timed region as
short as 20 steps of the default workload, 25 ms, holds samples."""
import os
import stat
import sys
import time

from conftest import ROOT

sys.path.insert(0, ROOT)

FAKE = """#!{python}
import sys, time
ms = float(sys.argv[sys.argv.index("-lms") + 1])
while True:
    print("1965, 1965, 500.0, 0x0, Not Active, Not Active, Not Active, Active", flush=True)
    time.sleep(ms / 1000)
"""


def test_short_region_is_sampled(tmp_path, monkeypatch):
    import bench
    exe = tmp_path / "nvidia-smi"
    exe.write_text(FAKE.format(python=sys.executable))
    exe.chmod(exe.stat().st_mode | stat.S_IXUSR)
    monkeypatch.setenv("PATH", str(tmp_path) + os.pathsep + os.environ["PATH"])
    for _ in range(3):  # a busy host may hold the stand-in up for a whole region
        with bench.ClockSampler(0) as s:
            time.sleep(0.025)
        got = s.summary()
        if got.get("samples"):
            break
    assert got.get("samples", 0) >= 1 and got["sm_mhz"] == 1965.0 and got["reasons"] == ["sw_power_cap"], got
