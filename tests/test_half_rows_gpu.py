"""The y transforms split into their even and odd rows (3D 32^3 and 64^3) are as accurate as the
unsplit ones: one step so long that the transformed products, not the rounding of the state,
make its error, in the split form and in the elementwise form, both against FP64."""
import numpy as np
import pytest

from oracle import numpy_ref as R

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from l3es import _native  # noqa: E402


@pytest.mark.parametrize("n,seeds", [(32, 8), (64, 4)])
def test_split_rows_lose_no_accuracy(n, seeds):
    nu, dt = 1e-3, 0.1
    step = R.rk4_wrapper(dt, R.rhs_wrapper(n, nu, (1, 2, 3)), None, 0.0, "none", (1, 2, 3))
    p = _native.Plan(dim=3, n=n, nu=nu, dt=dt)
    errs = {0: 0.0, 2: 0.0}
    for seed in range(seeds):
        u = R.init_u_hit(n, seed, spectrum="k4exp", kp=4.0)
        u = u * np.sqrt(0.5 / R.kinetic_energy(u))
        start = np.ascontiguousarray(np.fft.rfftn(u, axes=(1, 2, 3)), dtype=np.complex64)
        uh = start.astype(np.complex128)
        ref = step(np.fft.irfftn(uh, s=(n,) * 3, axes=(1, 2, 3)), uh)[1]
        for form in errs:
            p.step_form = form
            x = torch.from_numpy(start.copy()).cuda()
            p.step(x, 1)
            errs[form] += np.linalg.norm(x.cpu().numpy() - ref) ** 2 / np.linalg.norm(ref) ** 2 / seeds
    # the same radices, so the same errors but for their signs: sums of squares over more than
    # 10^5 modes, which low modes dominate, to 2 %
    assert np.sqrt(errs[2] / errs[0]) < 1.02, errs
