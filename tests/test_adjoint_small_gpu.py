"""The adjoint on the smallest grids, where the stored columns of the nonlinear term (kt, a
whole tile) reach or pass the half axis (N = 8: kt = 8, N/2 + 1 = 5): the RHS vector-Jacobian
product and the adjoint step against the FP64 oracle, 2D and 3D, one and two trajectories."""
import numpy as np
import pytest

from oracle import adjoint_ref as A
from oracle import numpy_ref as R

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from l3es import _native  # noqa: E402


def _c64(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.complex64)).cuda()


def _state(dim, n, seed):
    if dim == 3:
        u = R.init_u_hit(n, seed, "k4exp", 2.0)
        return np.fft.rfftn(u * np.sqrt(0.5 / R.kinetic_energy(u)), axes=(1, 2, 3))
    return np.fft.rfftn(R.init_u_random2d(n, seed, n / 4)[..., 0], axes=(1, 2))


def _check(dim, n, batch, forcing):
    nu, dt, kf = 5e-3, 2e-3, 2
    axes = (1, 2, 3) if dim == 3 else (1, 2)
    uh = np.stack([_state(dim, n, 3 + b) for b in range(batch)])
    rng = np.random.default_rng(n + dim)
    g = rng.standard_normal(uh.shape) + 1j * rng.standard_normal(uh.shape)
    if dim == 2:
        g[:, 2] = 0.0
    _, kkk2, _, _ = R.wavenumbers(n, dim)
    mask = ((kkk2 > 0) & (kkk2 <= kf * kf)).astype(float)
    cp = (0.1, mask) if forcing == "const_power" else None
    rhs = R.rhs_wrapper(n, nu, axes, const_power=cp)
    vjp = A.rhs_vjp_wrapper(n, nu, axes, const_power=cp)
    e_all = [A.ekin_tot_forward(u, mask, 0.0, n, dim) for u in uh]
    e0 = [0.95 * (e[2] + e[3]) for e in e_all]  # below the energy: the rescaling acts
    kw = {"const_power": dict(kf=kf, eps_inj=0.1), "ekin_tot": dict(kf=kf, e_kin_init=e0[0])}.get(forcing, {})
    p = _native.Plan(dim=dim, n=n, nu=nu, dt=dt, batch=batch, forcing=forcing, **kw)
    p.set_e0(e0)
    u, out = _c64(uh).reshape(p.spec_shape), _c64(uh).reshape(p.spec_shape)
    p.rhs_vjp(u, _c64(g).reshape(p.spec_shape), out)
    lam = _c64(g).reshape(p.spec_shape)
    p.adjoint_step(u, lam)
    for b in range(batch):
        ref = vjp(uh[b], g[b])
        end = g[b]
        if forcing == "ekin_tot":
            end = A.ekin_tot_vjp(A.rk4_step(uh[b], dt, rhs), g[b], mask, e0[b], n, dim)
        step = A.rk4_step_vjp(uh[b], end, dt, rhs, vjp)
        # 3e-5: the bound of the repository's adjoint tests (FP32 transforms)
        assert np.abs(out.cpu().numpy().reshape(uh.shape)[b] - ref).max() < 3e-5 * np.abs(ref).max(), b
        assert np.abs(lam.cpu().numpy().reshape(uh.shape)[b] - step).max() < 3e-5 * np.abs(step).max(), b


@pytest.mark.parametrize("forcing", ["none", "ekin_tot"])
@pytest.mark.parametrize("batch", [1, 2])
@pytest.mark.parametrize("n", [8, 16])
@pytest.mark.parametrize("dim", [2, 3])
def test_vjp_and_step_match_the_oracle(dim, n, batch, forcing):
    _check(dim, n, batch, forcing)


@pytest.mark.parametrize("batch", [1, 2])
@pytest.mark.parametrize("n", [8, 16])
@pytest.mark.parametrize("dim", [2, 3])
def test_constant_power_matches_the_oracle(dim, n, batch):
    """The band sums of blocks smaller than a warp (8 and 16 threads)."""
    _check(dim, n, batch, "const_power")


@pytest.mark.parametrize("dim,n", [(2, 8), (2, 16), (2, 32), (2, 64), (3, 8), (3, 16)])
def test_constant_power_rhs_of_small_blocks(dim, n):
    """The right-hand side's band coefficient by blocks of 4 to 16 threads (2D: tiles of 2 and
    of 8 columns)."""
    axes = (1, 2, 3) if dim == 3 else (1, 2)
    uh = _state(dim, n, 5)
    _, kkk2, _, _ = R.wavenumbers(n, dim)
    ref = R.rhs_wrapper(n, 5e-3, axes, const_power=(0.1, ((kkk2 > 0) & (kkk2 <= 4)).astype(float)))(None, uh, 1)
    p = _native.Plan(dim=dim, n=n, nu=5e-3, dt=1e-3, forcing="const_power", kf=2, eps_inj=0.1)
    for x_bulk in (1, 0):
        p.set_schedule({"x_bulk": x_bulk})
        u = _c64(uh)
        du = torch.empty_like(u)
        p.rhs(u, du)
        # 2e-5: the bound of the repository's step tests (FP32 transforms)
        assert np.abs(du.cpu().numpy() - ref).max() < 2e-5 * np.abs(ref).max(), x_bulk
