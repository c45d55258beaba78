"""The x forward pass that assembles the RHS vector-Jacobian product (3D from 64^3) against
the FP64 oracle: the smallest grid that takes it and the next with another thread count, two
trajectories, drag, the constant-power band, the product written over its own cotangent, and
the four chained stages of an adjoint step."""
import numpy as np
import pytest

from oracle import adjoint_ref as A
from oracle import numpy_ref as R

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from l3es import _native  # noqa: E402

AXES = (1, 2, 3)


def _c64(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.complex64)).cuda()


def _state(n, seed):
    u = R.init_u_hit(n, seed, "k4exp", 3.0)
    return np.fft.rfftn(u * np.sqrt(0.5 / R.kinetic_energy(u)), axes=AXES)


def _rel(a, b):
    return np.abs(a.cpu().numpy() - b).max() / np.abs(b).max()


@pytest.mark.parametrize("n,batch,drag,forced", [(64, 1, 0.1, False), (64, 2, 0.0, True), (128, 1, 0.05, True)])
def test_vjp_and_step_match_the_oracle(n, batch, drag, forced):
    nu, dt = 5e-3, 2e-3
    uh = np.stack([_state(n, 3 + b) for b in range(batch)])
    rng = np.random.default_rng(n)
    g = rng.standard_normal(uh.shape) + 1j * rng.standard_normal(uh.shape)
    cp = None
    if forced:
        _, kkk2, _, _ = R.wavenumbers(n, 3)
        cp = (0.1, ((kkk2 > 0) & (kkk2 <= 4)).astype(float))
    rhs = R.rhs_wrapper(n, nu, AXES, drag=drag, const_power=cp)
    vjp = A.rhs_vjp_wrapper(n, nu, AXES, drag=drag, const_power=cp)
    kw = dict(forcing="const_power", kf=2, eps_inj=0.1) if forced else {}
    p = _native.Plan(dim=3, n=n, nu=nu, dt=dt, drag=drag, batch=batch, **kw)
    shape = p.spec_shape
    u = _c64(uh).reshape(shape)
    out, same, lam = torch.empty_like(u), _c64(g).reshape(shape), _c64(g).reshape(shape)
    p.rhs_vjp(u, lam, out)
    p.rhs_vjp(u, same, same)
    assert torch.equal(out, same)
    p.adjoint_step(u, lam)
    for b in range(batch):
        # 3e-5: the bound of the repository's adjoint tests (FP32 transforms)
        assert _rel(out.reshape(uh.shape)[b], vjp(uh[b], g[b])) < 3e-5, b
        if n == 64:
            assert _rel(lam.reshape(uh.shape)[b], A.rk4_step_vjp(uh[b], g[b], dt, rhs, vjp)) < 3e-5, b
