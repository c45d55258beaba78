"""The exact spectral interpolation kernel at the edges of its split: particle counts around
a block's 16 or 32 particles and the change from one to the other, kx ranges smaller and
larger than the parts of a block. Against the FP64 sum over the same modes."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from l3es import _native  # noqa: E402


@pytest.mark.parametrize("dim,c,np_", [(3, 8, 1), (3, 8, 33), (3, 16, 17), (3, 32, 95), (3, 64, 31), (2, 8, 16),
                                       (2, 16, 32), (2, 32, 257), (2, 64, 63), (3, 8, 4864), (3, 8, 4865), (3, 16, 4897),
                                       (2, 8, 4881)])
def test_dft_interpolation_matches_the_sum(dim, c, np_):
    rng = np.random.default_rng(c + np_)
    u = rng.standard_normal((3,) + (c,) * dim).astype(np.float32)
    if dim == 2:
        u[2] = 0.0
    r = rng.uniform(0.0, 2 * np.pi, (np_, dim))
    dt = 0.3
    p = _native.InterpPlan(dim=dim, ckp_n=c, n_fine=0, np_max=np_)
    p.set_field(torch.from_numpy(u.reshape((3,) + (c,) * dim + ((1,) if dim == 2 else ()))).cuda())
    hh = torch.empty(p.coarse_spec_shape, dtype=torch.complex64, device="cuda")
    p.coarse_spectrum(hh)
    rt = torch.from_numpy(r).cuda()
    u_r, r_out = torch.empty_like(rt), torch.empty_like(rt)
    p.interp(rt, u_r, backend="dft", dt=dt, r_out=r_out)
    # full spectrum of the plan's own FP32 half spectrum: Hermitian below zero on the last axis
    h = hh.cpu().numpy().astype(np.complex128).reshape((3,) + (c,) * (dim - 1) + (c // 2 + 1,))
    full = np.zeros((3,) + (c,) * dim, dtype=np.complex128)
    full[..., : c // 2] = h[..., : c // 2]
    idx = (-np.arange(c)) % c
    for kz in range(1, c // 2 + 1):
        m = h[..., kz][:, idx]
        full[..., c - kz] = np.conj(m[:, :, idx] if dim == 3 else m)
    k = np.fft.fftfreq(c, 1.0 / c)
    ph = [np.exp(1j * r[:, d, None] * k) for d in range(dim)]
    if dim == 3:
        ref = np.einsum("fxyz,px,py,pz->pf", full, *ph, optimize=True)
    else:
        ref = np.einsum("fxy,px,py->pf", full, *ph, optimize=True)
    ref = ref.real[:, :dim] / c**dim
    # FP32 phases and a chain of 2c rounded FMAs per summed axis
    tol = dim * (2 * c + 4) * 2.0**-24 * np.abs(full[:dim]).reshape(dim, -1).sum(1) / c**dim
    assert np.all(np.abs(u_r.cpu().numpy() - ref) <= tol)
    moved = np.mod(r + dt * u_r.cpu().numpy(), 2 * np.pi)
    assert np.abs(r_out.cpu().numpy() - moved).max() <= 1e-12
