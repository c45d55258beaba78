"""The NUFFT's pruned grid passes and interleaved gather on every grid size, width and
dimension, single and batched, against the exact sum over the same modes (the library's
FP64-checked dft backend, plan by plan)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from l3es import _native  # noqa: E402


@pytest.mark.parametrize("dim,c,width,np_,batch", [
    (3, 8, 6, 1, 1), (3, 16, 8, 37, 1), (3, 32, 6, 1001, 2), (3, 64, 4, 130, 1), (2, 8, 6, 5, 3), (2, 16, 4, 33, 1),
    (2, 32, 8, 129, 1), (2, 64, 6, 64, 2)])
def test_nufft_matches_the_exact_sum(dim, c, width, np_, batch):
    rng = np.random.default_rng(7 * c + width)
    n = c
    axes = tuple(range(2, 2 + dim))
    u = rng.standard_normal((batch, 3) + (n,) * dim)
    uh = torch.from_numpy(np.fft.rfftn(u, axes=axes).astype(np.complex64)).cuda()
    # positions on the box's edges among them
    r = rng.uniform(0.0, 2 * np.pi, (batch, np_, dim))
    r[:, 0] = 0.0
    r[:, -1] = np.nextafter(2 * np.pi, 0.0)
    rt = torch.from_numpy(r).cuda()
    got, moved = torch.empty_like(rt), torch.empty_like(rt)
    p = _native.InterpPlan(dim=dim, ckp_n=c, n_fine=n, width=width, np_max=np_, batch=batch)
    if batch == 1:
        p.set_spectrum(uh[0].contiguous())
        p.interp(rt[0], got[0], dt=0.25, r_out=moved[0])
    else:
        p.set_spectrum(uh)
        p.interp(rt, got, dt=0.25, r_out=moved)
    one = _native.InterpPlan(dim=dim, ckp_n=c, n_fine=n, np_max=np_)
    ref = torch.empty_like(rt)
    for b in range(batch):
        one.set_spectrum(uh[b].contiguous())
        one.interp(rt[b], ref[b], backend="dft")
    # the kernel of width w has an error of about 10^(1 - w) per axis; FP32 grids end near 1e-6
    tol = dim * max(2.0 * 10.0 ** (1 - width), 2e-6)
    assert (got - ref).norm() <= tol * ref.norm()
    want = np.mod(r + 0.25 * got.cpu().numpy(), 2 * np.pi)
    d = np.abs(moved.cpu().numpy() - want)
    assert np.minimum(d, 2 * np.pi - d).max() <= 1e-12
