"""GPU: spanwise lengths that are odd (27, 81 points): the two rows that share a
streamwise transform may lie in different planes, in a batch of different members.

The FP64 step against the oracle at the parity bar of the step, 1e-11, after two
steps; a batch bit for bit its members as separate contexts; the reference-layout
transforms at theirs, 1e-13 of the largest value (486 and 27 points: streamwise
lengths without a plan)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import rpcf_oracle as O  # noqa: E402


@pytest.fixture(autouse=True)
def _need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("mx,my,mz", [(24, 27, 32), (48, 81, 32), (27, 27, 36)])
def test_step_matches_oracle(pkg, mx, my, mz):
    kw = dict(Re=1300.0, Ro=0.3, dt=0.002)
    c = pkg.Context(pkg.make_params(mx, my, mz, **kw))
    pb = O.Problem(O.Params(mx, my, mz, prof=(0.5, 0.5, 0.0), **kw))
    s = pkg.seeded_state(c.Nx, c.Ny, c.Nz, amplitude=0.05, seed=3)
    c.set_state(*s)
    pb.set_state(*s)
    c.bootstrap()
    pb.bootstrap()
    for _ in range(2):
        c.step(1)
        pb.step()
    for got, ref in zip(c.get_state(), (pb.V, pb.O)):
        assert np.linalg.norm(got - ref) < 1e-11 * np.linalg.norm(ref)
    c.close()


def test_batch_equals_members(pkg):
    mx, my, mz = 24, 27, 32
    runs = [dict(Re=500.0, Ro=0.0, dt=0.002), dict(Re=1300.0, Ro=0.3, dt=0.001), dict(Re=3000.0, Ro=0.1, dt=0.004)]
    ps = [pkg.make_params(mx, my, mz, **r) for r in runs]
    b = pkg.BatchContext(ps)
    states = [pkg.seeded_state(b.Nx, b.Ny, b.Nz, amplitude=0.05, seed=k) for k in range(len(ps))]
    b.set_state(*(np.stack([s[i] for s in states]) for i in range(2)))
    b.bootstrap()
    b.step(2)
    got = b.get_state()
    for k, p in enumerate(ps):
        c = pkg.Context(p)
        c.set_state(*states[k])
        c.bootstrap()
        c.step(2)
        assert all(np.array_equal(got[i][k], x) for i, x in enumerate(c.get_state())), k
        c.close()
    b.close()


@pytest.mark.parametrize("mx,my,mz", [(24, 27, 32), (27, 27, 32), (486, 27, 16), (48, 81, 64)])
def test_transform_matches_oracle(pkg, mx, my, mz):
    sz = O.Sizes(mx, my, mz)
    r = np.random.default_rng(mx + my)
    S = np.zeros((sz.ny, sz.hnx, mz), dtype=np.complex128)
    S[..., :sz.nz] = r.standard_normal((sz.ny, sz.hnx, sz.nz)) + 1j * r.standard_normal((sz.ny, sz.hnx, sz.nz))
    pitch = (mx // 2 + 1) * 16
    c = pkg.Context(pkg.make_params(mx, my, mz, Re=1300.0, dt=0.001))
    spec = torch.from_numpy(S).cuda()
    phys = torch.zeros(sz.pz, my, pitch // 8, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    c.transform_3d_one(pkg.BACKWARD, phys.data_ptr(), pitch, spec.data_ptr(), mz * 16)
    c.synchronize()
    ref = O.transform_backward(S, sz)
    assert np.abs(phys.cpu().numpy()[..., :mx] - ref).max() < 1e-13 * np.abs(ref).max()
    P = r.standard_normal((sz.pz, my, mx))
    phys[..., :mx] = torch.from_numpy(P)
    torch.cuda.synchronize()
    c.transform_3d_one(pkg.FORWARD, phys.data_ptr(), pitch, spec.data_ptr(), mz * 16)
    c.synchronize()
    ref = O.transform_forward(P, sz)[..., :sz.pz]
    assert np.abs(spec.cpu().numpy()[..., :sz.pz] - ref).max() < 1e-13 * np.abs(ref).max()
    c.close()
