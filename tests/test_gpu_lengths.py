"""GPU: every line length with a compiled transform, in both precisions.

The passes along each direction exist per length (2^a 3^b); grids that are
short in the other two directions put every length through the drop-in
transforms (FP64, against the oracle: 1e-13 of the largest value, the parity
bar of the transforms) and through the time step (the mixed form against FP64:
1e-6 relative after two steps, the bar of the variants; the FP64 streamwise
and wall-normal passes against their block forms: 1e-12, and 1e-11, the step's
parity bar, where the two forms build the right-hand sides differently).  The short directions leave ragged tiles:
9 streamwise modes, 17 wall-normal points, 54 span points (no multiple of 4)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import rpcf_oracle as O  # noqa: E402

SPAN = [24, 32, 36, 48, 54, 64, 72, 96, 108, 128, 144, 162, 192, 216, 256, 288, 324, 384, 432, 512, 576, 768]
WALL = [32, 36, 48, 64, 72, 96, 108, 128, 144, 192, 216, 256, 288, 324, 384, 432, 512, 576, 768]


@pytest.fixture(autouse=True)
def _need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _transform_errors(pkg, mx, my, mz):
    sz = O.Sizes(mx, my, mz)
    r = np.random.default_rng(mx * 7 + my * 3 + mz)
    S = np.zeros((sz.ny, sz.hnx, mz), dtype=np.complex128)
    S[..., :sz.nz] = r.standard_normal((sz.ny, sz.hnx, sz.nz)) + 1j * r.standard_normal((sz.ny, sz.hnx, sz.nz))
    pitch = (mx // 2 + 1) * 16
    c = pkg.Context(pkg.make_params(mx, my, mz, Re=1300.0, dt=0.001))
    spec = torch.from_numpy(S).cuda()
    phys = torch.zeros(sz.pz, my, pitch // 8, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    c.transform_3d_one(pkg.BACKWARD, phys.data_ptr(), pitch, spec.data_ptr(), mz * 16)
    c.synchronize()
    got = phys.cpu().numpy()[..., :mx]
    ref = O.transform_backward(S, sz)
    eb = np.abs(got - ref).max() / np.abs(ref).max()
    P = r.standard_normal((sz.pz, my, mx))
    phys[..., :mx] = torch.from_numpy(P)
    torch.cuda.synchronize()
    c.transform_3d_one(pkg.FORWARD, phys.data_ptr(), pitch, spec.data_ptr(), mz * 16)
    c.synchronize()
    got = spec.cpu().numpy()[..., :sz.pz]
    ref = O.transform_forward(P, sz)[..., :sz.pz]
    ef = np.abs(got - ref).max() / np.abs(ref).max()
    c.close()
    return eb, ef


def _state_after(pkg, prec, mx, my, mz, variants=(), U=(0.5, 0.5, 0.0)):
    c = pkg.Context(pkg.make_params(mx, my, mz, Re=1300.0, Ro=0.1, dt=0.001, U=U, precision=prec))
    for p, v in variants:
        c.set_variant(p, v)
    c.set_state(*pkg.seeded_state(c.Nx, c.Ny, c.Nz, amplitude=0.05, seed=1))
    c.bootstrap()
    c.step(2)
    out = c.get_state()
    c.close()
    return out


def _apart(x, y):
    return max(np.linalg.norm(a - b) / np.linalg.norm(b) for a, b in zip(x, y))


def _step_error(pkg, mx, my, mz, variants=()):
    return _apart(_state_after(pkg, pkg.PREC_MIXED, mx, my, mz, variants), _state_after(pkg, pkg.PREC_FP64, mx, my, mz))


@pytest.mark.parametrize("L", SPAN)
def test_span_length(pkg, L):
    eb, ef = _transform_errors(pkg, 24, L, 32)
    assert eb < 1e-13 and ef < 1e-13, (eb, ef)
    e = _step_error(pkg, 24, L, 32, [(pkg.PASS_ZB, pkg.Z_WARP), (pkg.PASS_ZF, pkg.Z_WARP)])
    assert e < 1e-6, e


@pytest.mark.parametrize("L", SPAN)
def test_stream_length(pkg, L):
    fused = _state_after(pkg, pkg.PREC_FP64, L, 54, 32)
    block = _state_after(pkg, pkg.PREC_FP64, L, 54, 32, [(pkg.PASS_X, pkg.X_BLOCK)])
    assert _apart(fused, block) < 1e-12
    e = _step_error(pkg, L, 54, 32, [(pkg.PASS_X, pkg.X_WARP3)])
    assert e < 1e-6, e


@pytest.mark.parametrize("M", WALL)
def test_wall_length(pkg, M):
    eb, ef = _transform_errors(pkg, 24, 24, M)
    assert eb < 1e-13 and ef < 1e-13, (eb, ef)
    warp, block = [(pkg.PASS_Y3, pkg.Y3_FFT)], [(pkg.PASS_Y3, pkg.Y3_BLOCK)]
    assert _apart(*(_state_after(pkg, pkg.PREC_FP64, 24, 24, M, v) for v in (warp, block))) < 1e-12
    warp, block = [(pkg.PASS_Y1, pkg.Y1_WARP)], [(pkg.PASS_Y1, pkg.Y1_BLOCK)]
    for U in ((0.5, 0.5, 0.0), (1.0, 0.0, -1.0), (0.3, 0.7, -0.4)):
        assert _apart(*(_state_after(pkg, pkg.PREC_FP64, 24, 24, M, v, U) for v in (warp, block))) < 1e-11, U
    e = _step_error(pkg, 24, 24, M, [(pkg.PASS_Y3, pkg.Y3_FFT), (pkg.PASS_Y1, pkg.Y1_WARP)])
    assert e < 1e-6, e


@pytest.mark.parametrize("M", WALL)
def test_cheby_whole_line(pkg, M):
    """dns_cheby_s2p / p2s fill the FFT's whole line, as the reference does in place."""
    sz = O.Sizes(24, 24, M)
    r = np.random.default_rng(M)
    c = pkg.Context(pkg.make_params(24, 24, M, Re=1300.0, dt=0.001))
    for pad in (pkg.PADDING, pkg.NO_PADDING):
        line = M if pad == pkg.PADDING else M // 2
        for f, ref in ((c.cheby_s2p, O.cheby_s2p), (c.cheby_p2s, O.cheby_p2s)):
            S = r.standard_normal((sz.ny, sz.hnx, M)) + 1j * r.standard_normal((sz.ny, sz.hnx, M))
            t = torch.from_numpy(S).cuda()
            torch.cuda.synchronize()
            f(t.data_ptr(), M * 16, pad)
            c.synchronize()
            got, exp = t.cpu().numpy(), ref(S, M, pad == pkg.PADDING)
            assert np.abs(got[..., :line] - exp[..., :line]).max() < 1e-13 * np.abs(exp[..., :line]).max()
            assert np.array_equal(got[..., line:], S[..., line:])
    c.close()


@pytest.mark.parametrize("mx,my,mz", [(24, 24, 32), (96, 192, 256)])
def test_six_fields_equal_one_by_one(pkg, mx, my, mz):
    """dns_transform shares launches between fields (the second grid's rows
    fill the workspace with two): bit for bit the fields one by one."""
    sz = O.Sizes(mx, my, mz)
    pitch = (mx // 2 + 1) * 16
    g = torch.Generator(device="cuda").manual_seed(5)
    c = pkg.Context(pkg.make_params(mx, my, mz, Re=1300.0, dt=0.001))
    spec = [torch.randn(sz.ny, sz.hnx, mz, dtype=torch.complex128, device="cuda", generator=g) for _ in range(6)]
    out = []
    for together in (True, False):
        s = [t.clone() for t in spec]
        p = [torch.zeros(sz.pz, my, pitch // 8, dtype=torch.float64, device="cuda") for _ in s]
        torch.cuda.synchronize()
        for d in (pkg.BACKWARD, pkg.FORWARD):
            groups = [range(6)] if together else [[i] for i in range(6)]
            for i in groups:
                c.transform(d, [p[k].data_ptr() for k in i], pitch, [s[k].data_ptr() for k in i], mz * 16)
        c.synchronize()
        out.append([t.cpu().numpy()[..., :mx] for t in p] + [t.cpu().numpy()[..., :sz.pz] for t in s])
    assert all(np.array_equal(a, b) for a, b in zip(*out))
    c.close()


@pytest.mark.parametrize("M", [36, 64, 108, 128, 256])
def test_solve_one_system(pkg, M):
    """dns_solve_wall of one system (36, 108: no DCT plan for 2 (Ny - 1) points)
    equals that system of a call with both, bit for bit, and leaves no other."""
    sz = O.Sizes(24, 24, M)
    g = torch.Generator(device="cuda").manual_seed(M)
    b = [torch.randn(sz.ny, sz.hnx, M, dtype=torch.complex128, device="cuda", generator=g) for _ in range(2)]
    c = pkg.Context(pkg.make_params(24, 24, M, Re=1300.0, dt=0.001))
    both, one = [t.clone() for t in b], [t.clone() for t in b]
    torch.cuda.synchronize()
    c.solve_wall(both[0].data_ptr(), both[1].data_ptr(), M * 16)
    c.solve_wall(one[0].data_ptr(), None, M * 16)
    c.solve_wall(None, one[1].data_ptr(), M * 16)
    for x, y, z in zip(both, one, b):
        assert torch.equal(x, y)
        assert torch.equal(x[..., sz.nz:], z[..., sz.nz:])
    c.close()


@pytest.mark.parametrize("mz", [128, 108])  # a wall-normal length with a plan, one without
@pytest.mark.parametrize("offset", [0, 8])
def test_history_on_device_pointers(pkg, mz, offset):
    """The AB2 history to and from device pencils of a wider pitch, 16- and 8-byte
    aligned, against the host form: the same kernel on the same values."""
    c = pkg.Context(pkg.make_params(24, 24, mz, Re=1300.0, dt=0.001))
    r = np.random.default_rng(3)
    V, W = (r.standard_normal(c.shape) + 1j * r.standard_normal(c.shape) for _ in range(2))
    c.set_history(V, W)
    hv, ho = c.get_history()
    H, Ny = int(np.prod(c.shape[:-1])), c.shape[-1]
    row = 2 * Ny + 6  # doubles per pencil
    buf = [torch.zeros(H * row + 1, dtype=torch.float64, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    ptr = [b.data_ptr() + offset for b in buf]
    view = [b[offset // 8:offset // 8 + H * row].view(H, row)[:, :2 * Ny] for b in buf]
    c._call("dns_get_history", ptr[0], ptr[1], row * 8, pkg.DEVICE)
    for a, b in zip(view, (hv, ho)):
        assert np.array_equal(a.cpu().numpy(), np.ascontiguousarray(b).view(np.float64).reshape(H, 2 * Ny))
    c.set_history(W, V)
    c._call("dns_set_history", ptr[0], ptr[1], row * 8, pkg.DEVICE)
    c2 = pkg.Context(pkg.make_params(24, 24, mz, Re=1300.0, dt=0.001))
    c2.set_history(hv, ho)
    for a, b in zip(c.get_history(), c2.get_history()):
        assert np.array_equal(a, b)
