"""Diagnostics on the grids where their tilings can go wrong: the smallest and odd-sized
shares per thread, 2D and 3D, batched, and fields that hold infinities or NaN."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from l3es import _native  # noqa: E402


def _spec(dim, n, batch, seed):
    u = np.random.default_rng(seed).standard_normal((batch, 3) + (n,) * dim).astype(np.float32)
    return u, np.fft.rfftn(u, axes=tuple(range(2, 2 + dim))).astype(np.complex64)


@pytest.mark.parametrize("dim,n,batch", [(3, 8, 1), (3, 16, 3), (3, 64, 1), (2, 8, 2), (2, 32, 1), (2, 128, 2)])
def test_diagnostics_match_fp64_sums(dim, n, batch):
    u, uh = _spec(dim, n, batch, n + dim)
    p = _native.Plan(dim=dim, n=n, nu=1e-2, dt=1e-3, batch=batch)
    ut = torch.from_numpy(u.reshape((batch, 3) + (n,) * dim + ((1,) if dim == 2 else ()))).cuda()
    ht = torch.from_numpy(uh).cuda()
    if batch == 1:
        ut, ht = ut[0].contiguous(), ht[0].contiguous()
    ek = torch.empty(batch * n, dtype=torch.float64, device="cuda")
    st = torch.empty(batch * 4, dtype=torch.float64, device="cuda")
    eps = torch.empty(batch, dtype=torch.float64, device="cuda")
    p.energy_spectrum(ht, ek)
    p.field_stats(ut, st)
    p.dissipation(ht, 1e-2, eps)
    k = np.fft.fftfreq(n, 1.0 / n)
    kh = np.arange(n // 2 + 1.0)
    g = np.meshgrid(*([k] * (dim - 1)), kh, indexing="ij")
    kk = np.stack([g[0], g[1], g[2] if dim == 3 else np.zeros_like(g[0])])
    w = np.where((kh == 0) | (kh == n // 2), 1.0, 2.0) * np.ones_like(g[0])
    shell = (np.sqrt((kk**2).sum(0)) + 0.5).astype(int).ravel()
    for b in range(batch):
        h = uh[b].astype(np.complex128)
        e = w * (np.abs(h) ** 2).sum(0) / float(n) ** (2 * dim)
        cnt = np.bincount(shell, w.ravel(), minlength=n)[:n]
        tot = np.bincount(shell, e.ravel(), minlength=n)[:n]
        kr = np.arange(n)
        ref = tot * 4 * np.pi * kr**2 / (cnt + np.finfo(float).eps)
        # each mode's energy is formed by 6 FP32 FMAs
        assert np.all(np.abs(ek.cpu().numpy()[b * n:(b + 1) * n] - ref) <= 6 * 2.0**-24 * ref + 1e-300)
        f = u[b].astype(np.float64)
        s = st.cpu().numpy()[4 * b:4 * b + 4]
        assert np.array_equal(s[:3], np.abs(f).reshape(3, -1).max(1))
        assert abs(s[3] - 0.5 * (f * f).sum(0).mean()) <= 3 * 2.0**-24 * s[3]
        c = 1j * np.cross(kk, h, axis=0)
        om = np.fft.irfftn(c, s=(n,) * dim, axes=tuple(range(1, 1 + dim)))
        ref_eps = 1e-2 * (om * om).sum(0).mean()
        assert abs(eps.cpu().numpy()[b] - ref_eps) <= 16 * 2.0**-24 * ref_eps


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan, 3e19])
def test_field_stats_and_spectrum_of_bad_values(bad):
    """What a blow-up shows in the log columns: an infinite or overflowing value gives an
    infinite energy, a NaN a NaN."""
    n = 16
    u, uh = _spec(3, n, 1, 1)
    u[0, 1, 3, 4, 5] = bad
    uh[0, 2, 1, 2, 3] = bad
    p = _native.Plan(dim=3, n=n, nu=1e-2, dt=1e-3)
    st = torch.empty(4, dtype=torch.float64, device="cuda")
    ek = torch.empty(n, dtype=torch.float64, device="cuda")
    p.field_stats(torch.from_numpy(u[0]).cuda(), st)
    p.energy_spectrum(torch.from_numpy(uh[0]).cuda(), ek)
    same = np.isnan if np.isnan(bad) else np.isposinf
    assert same(st.cpu().numpy()[3]) and same(ek.cpu().numpy()[int(np.sqrt(14) + 0.5)])


def test_dissipation_and_stats_of_misaligned_arrays():
    """The C entry points take spectra and fields at any element's address; the kernels load
    16 bytes at a time where the address allows it."""
    n = 32
    u, uh = _spec(3, n, 1, 4)
    p = _native.Plan(dim=3, n=n, nu=1e-2, dt=1e-3)
    lib, s = p._lib, torch.cuda.current_stream().cuda_stream
    got = []
    for shift in (0, 1):
        hb = torch.zeros(uh.size + 2, dtype=torch.complex64, device="cuda")
        hb[shift:shift + uh.size] = torch.from_numpy(uh.ravel()).cuda()
        fb = torch.zeros(u.size + 4, dtype=torch.float32, device="cuda")
        fb[shift:shift + u.size] = torch.from_numpy(u.ravel()).cuda()
        out = torch.empty(5, dtype=torch.float64, device="cuda")
        assert lib.l3es_dissipation(p._h, hb.data_ptr() + 8 * shift, 1e-2, out.data_ptr(), s) == 0
        assert lib.l3es_field_stats(p._h, fb.data_ptr() + 4 * shift, out.data_ptr() + 8, s) == 0
        got.append(out.cpu().numpy())
    assert np.array_equal(got[0], got[1])
