"""The x pass that closes an RK stage and opens the next one (kx_stage) against the FP64
oracle's RK4 steps, at the edges of where the step takes it: the smallest grids (fewer
threads per component than a warp), partly filled column tiles, 64^3 at the largest batch
that takes it and one above, several steps in one call (the new state's inverse transform
inside the last stage) and the forcings whose coefficient or rescale sits between stages."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from l3es import _native  # noqa: E402
from oracle import numpy_ref as R  # noqa: E402

STEPS = 3
# FP32 step against FP64, relative to the largest mode: the bound of the repository's step tests
RTOL = 2e-5


def _initial(dim, n, seed):
    if dim == 2:
        return R.init_u_random2d(n, seed, min(8.0, n / 4))
    u = R.init_u_hit(n, seed, spectrum="k4exp", kp=3.0)
    return u * np.sqrt(0.5 / R.kinetic_energy(u))


@pytest.mark.parametrize("dim,n,batch,forcing", [
    (3, 16, 1, "const_power"), (3, 32, 2, "none"), (3, 32, 1, "ekin_tot"), (3, 64, 4, "const_power"),
    (3, 64, 5, "none"), (2, 16, 3, "kolmogorov"), (2, 32, 1, "const_power"), (2, 64, 1, "ekin_tot"),
    (2, 128, 2, "kolmogorov"), (2, 512, 1, "kolmogorov"),
    (2, 256, 1, "kolmogorov"), (2, 256, 4, "none"), (2, 256, 5, "none"),
    (3, 64, 1, "const_power"), (3, 64, 2, "none"), (3, 32, 3, "none")])
def test_steps_match_the_oracle(dim, n, batch, forcing):
    axes = (1, 2, 3) if dim == 3 else (1, 2)
    nu, dt, drag = 5e-3, 2e-3 if dim == 3 else 1e-3, 0.1 if forcing == "kolmogorov" else 0.0
    kw, ref_kw = {}, {}
    if forcing == "const_power":
        kw = ref_kw = dict(forcing="const_power", kf=2, eps_inj=0.1)
    elif forcing == "ekin_tot":
        kw = dict(forcing="ekin_tot", kf=2, e_kin_init=0.5)
    elif forcing == "kolmogorov":
        kw = dict(drag=drag, kolm_k=4 if n > 16 else 2, kolm_amp=1.0)
    us = [_initial(dim, n, 5 + b) for b in range(batch)]
    uh0 = np.stack([np.fft.rfftn(u, axes=axes).reshape((3,) + (n,) * (dim - 1) + (n // 2 + 1,)) for u in us])
    p = _native.Plan(dim=dim, n=n, nu=nu, dt=dt, batch=batch, **kw)
    uh = torch.from_numpy(np.ascontiguousarray(uh0 if batch > 1 else uh0[0], dtype=np.complex64)).cuda()
    p.step(uh, STEPS)
    p.check()
    got = uh.cpu().numpy().reshape(uh0.shape)
    p.step_form = 0  # the elementwise update of the whole spectrum
    uh2 = torch.from_numpy(np.ascontiguousarray(uh0 if batch > 1 else uh0[0], dtype=np.complex64)).cuda()
    p.step(uh2, STEPS)
    plain = uh2.cpu().numpy().reshape(uh0.shape)
    assert np.abs(got - plain).max() <= 2e-6 * np.abs(plain).max()
    if forcing == "const_power" or (dim == 3 and n == 64):
        return  # the elementwise form is the reference (pinned to the oracle elsewhere)
    rhs = R.rhs_wrapper(n, nu, axes, drag=drag, force_hat=R.kolmogorov_forcing_hat(n, 1.0, kw["kolm_k"])) \
        if forcing == "kolmogorov" else R.rhs_wrapper(n, nu, axes)
    if forcing == "ekin_tot":
        step = R.rk4_wrapper(dt, rhs, R.init_forcing_mask_hit(n, 2) if dim == 3 else _mask2d(n, 2), 0.5, "ekin_tot", axes)
    else:
        step = R.rk4_wrapper(dt, rhs, None, 0.0, "none", axes)
    for b in range(batch):
        u, h = us[b], uh0[b]
        for _ in range(STEPS):
            u, h, _ = step(u, h)
        assert np.abs(got[b] - h).max() <= RTOL * np.abs(h).max(), b


def _mask2d(n, kf):
    k = np.fft.fftfreq(n, 1.0 / n)
    k2 = k[:, None] ** 2 + np.arange(n // 2 + 1)[None, :] ** 2
    return ((k2 > 0) & (k2 <= kf * kf)).astype(float)
