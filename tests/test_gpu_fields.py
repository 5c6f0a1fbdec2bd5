"""GPU: dns_transform on fields that share memory goes field by field, in order:
bit for bit the same calls one at a time."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import rpcf_oracle as O  # noqa: E402


@pytest.fixture(autouse=True)
def _need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("direction", ["backward", "forward"])
def test_two_fields_one_output(pkg, direction):
    mx, my, mz = 48, 48, 64
    sz = O.Sizes(mx, my, mz)
    pitch = (mx // 2 + 1) * 16
    c = pkg.Context(pkg.make_params(mx, my, mz, Re=1300.0, dt=0.001))
    g = torch.Generator(device="cuda").manual_seed(9)
    spec = [torch.randn(sz.ny, sz.hnx, mz, dtype=torch.complex128, device="cuda", generator=g) for _ in range(3)]
    phys = [torch.randn(sz.pz, my, pitch // 8, dtype=torch.float64, device="cuda", generator=g) for _ in range(3)]
    d = pkg.BACKWARD if direction == "backward" else pkg.FORWARD
    # the first and the last field have one output
    p_of, s_of = ([0, 1, 0], [0, 1, 2]) if direction == "backward" else ([0, 1, 2], [0, 1, 0])
    out = []
    for together in (True, False):
        s, p = [t.clone() for t in spec], [t.clone() for t in phys]
        torch.cuda.synchronize()
        for i in [[0, 1, 2]] if together else [[0], [1], [2]]:
            c.transform(d, [p[p_of[k]].data_ptr() for k in i], pitch, [s[s_of[k]].data_ptr() for k in i], mz * 16)
        c.synchronize()
        out.append([t.cpu().numpy() for t in s + p])
    assert all(np.array_equal(a, b) for a, b in zip(*out))
    c.close()
