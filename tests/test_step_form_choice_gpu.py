"""A 2D plan's step form: what it reports and takes before any is set, and that setting 1
selects the elementwise update (its kernels, and steps that agree with the other forms)."""
import numpy as np
import pytest

from oracle import numpy_ref as R

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from l3es import _native  # noqa: E402


@pytest.mark.parametrize("n", [16, 32, 64, 256])
def test_form_one_is_the_elementwise_update_in_2d(n):
    p = _native.Plan(dim=2, n=n, nu=5e-3, dt=1e-3, drag=0.1, kolm_k=2, kolm_amp=1.0)
    uh = torch.from_numpy(np.fft.rfftn(R.init_u_random2d(n, 3, n / 8)[..., 0], axes=(1, 2)).astype(np.complex64)).cuda()

    def run():
        x = uh.clone()
        p.timing(True)
        p.step(x, 3)
        names = set(p.kernel_stats())
        p.timing(False)
        return x, names

    start, kernels = run()
    assert p.step_form == 1 and "kx_stage" in kernels and "rk_update" not in kernels
    outs = {}
    for form in (2, 1, 0):
        p.step_form = form
        assert p.step_form == form
        outs[form], kernels = run()
        assert ("rk_update" in kernels) == (form < 2) and ("kx_stage" in kernels) == (form == 2), form
    assert torch.equal(outs[2], start)
    for form in (1, 0):
        # FP32 rounding: the bound of the repository's tests of the forms
        assert float((outs[form] - start).abs().max()) < 2e-6 * float(start.abs().max()), form
