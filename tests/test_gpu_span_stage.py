"""GPU: the tensor-staged spanwise passes of the mixed form at every length
that takes them, lengths that are no multiple of 16 among them.

Against the FP64 step 1e-6 relative after two steps, the bar of the variants.
9 streamwise modes and 17 wall-normal points leave ragged tiles."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# every spanwise length with a plan whose second radix fits half a warp
STAGED = [24, 32, 36, 48, 54, 64, 72, 96, 108, 128, 144, 162, 192, 216, 256, 288, 384, 512]


@pytest.fixture(autouse=True)
def _need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _state_after(pkg, prec, my, passes=()):
    c = pkg.Context(pkg.make_params(24, my, 32, Re=1300.0, Ro=0.1, dt=0.001, precision=prec))
    for p in passes:
        c.set_variant(p, pkg.Z_TENSOR_COPY)
    c.set_state(*pkg.seeded_state(c.Nx, c.Ny, c.Nz, amplitude=0.05, seed=1))
    c.bootstrap()
    c.step(2)
    out, chosen = c.get_state(), [c.get_variant(p) for p in (pkg.PASS_ZB, pkg.PASS_ZF)]
    c.close()
    return out, chosen


def _apart(x, y):
    return max(np.linalg.norm(a - b) / np.linalg.norm(b) for a, b in zip(x, y))


@pytest.mark.parametrize("L", STAGED)
def test_staged_length(pkg, L):
    ref, _ = _state_after(pkg, pkg.PREC_FP64, L)
    passes = [pkg.PASS_ZF] + ([pkg.PASS_ZB] if L <= 384 else [])  # the inverse stages Nz <= 256 modes
    got, chosen = _state_after(pkg, pkg.PREC_MIXED, L, passes)
    assert chosen[1] == pkg.Z_TENSOR_COPY
    assert _apart(got, ref) < 1e-6
    got, chosen = _state_after(pkg, pkg.PREC_MIXED, L)  # what a context takes by itself
    assert (chosen[1] == pkg.Z_TENSOR_COPY) == (L >= 144)
    assert _apart(got, ref) < 1e-6
