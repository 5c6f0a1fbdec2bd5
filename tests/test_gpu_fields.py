"""GPU: the buffers of dns_transform.

Fields that share memory go field by field, in order: bit for bit the same calls
one at a time.  A call takes no more row buffer than its fields need."""
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


def test_row_buffer(pkg):
    """Histories through host buffers take none, a call of one field that field's
    rows, a call of six their own; the results do not depend on it."""
    mx, my, mz = 48, 48, 64
    sz = O.Sizes(mx, my, mz)
    pitch = (mx // 2 + 1) * 16
    one = sz.pz * my * -(-(mx // 2 + 1) // 8) * 8 * 16  # rows of mx/2 + 1 bins rounded up to 8
    c = pkg.Context(pkg.make_params(mx, my, mz, Re=1300.0, dt=0.001))
    start = c.memory_bytes()
    r = np.random.default_rng(1)
    V, W = (r.standard_normal(c.shape) + 1j * r.standard_normal(c.shape) for _ in range(2))
    c.set_history(V, W)
    hv, ho = c.get_history()
    for got, x in ((hv, V), (ho, W)):  # there and back: ten times the parity bar of one transform
        assert np.abs(got - x).max() < 1e-12 * np.abs(x).max()
    assert c.memory_bytes() == start
    g = torch.Generator(device="cuda").manual_seed(4)
    spec = [torch.randn(sz.ny, sz.hnx, mz, dtype=torch.complex128, device="cuda", generator=g) for _ in range(6)]
    out = []
    for nf in (1, 6, 1):
        s = [t.clone() for t in spec]
        p = [torch.zeros(sz.pz, my, pitch // 8, dtype=torch.float64, device="cuda") for _ in s]
        torch.cuda.synchronize()
        for f in range(0, 6, nf):
            c.transform(pkg.BACKWARD, [t.data_ptr() for t in p[f:f + nf]], pitch,
                        [t.data_ptr() for t in s[f:f + nf]], mz * 16)
        c.synchronize()
        out.append([t.cpu().numpy()[..., :mx] for t in p])
        assert c.memory_bytes() == start + one * (1 if len(out) == 1 else 7)
    for x in out[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(x, out[0]))
    c.close()
