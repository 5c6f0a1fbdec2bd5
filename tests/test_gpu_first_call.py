"""GPU: the first call of a process loads the device code that it runs, not all
passes, lengths and precisions of the library.

The first bootstrap of a new process, best of three: 4 ms in FP64 and 7 to 10 in
the mixed form, against 34 with all passes of both in two modules; 20 lies
between."""
import os
import subprocess
import sys

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from conftest import ROOT  # noqa: E402

CHILD = """
import sys, time
sys.path.insert(0, {root!r} + "/tests")
from conftest import load_package
pkg = load_package()
c = pkg.Context(pkg.make_params(96, 96, 128, Re=1300.0, dt=0.001, precision={prec}))
c.set_state(*pkg.seeded_state(c.Nx, c.Ny, c.Nz, amplitude=0.05, seed=1))
c.synchronize()
t = time.perf_counter()
c.bootstrap()
c.synchronize()
print(time.perf_counter() - t)
"""


@pytest.mark.parametrize("prec", [0, 1])
def test_first_bootstrap_of_a_process(prec):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    times = []
    for _ in range(3):
        r = subprocess.run([sys.executable, "-c", CHILD.format(root=ROOT, prec=prec)], capture_output=True, text=True,
                           timeout=120, cwd=os.path.join(ROOT, "tests"))
        assert r.returncode == 0, r.stderr[-2000:]
        times.append(float(r.stdout.split()[-1]))
    assert min(times) < 0.020, times
