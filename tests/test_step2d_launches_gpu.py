"""Long runs of the small 2D grids whose steps share a launch: no launch takes the whole run,
the runs agree with the same steps in several calls to the bit, every step's e_inj is written."""
import numpy as np
import pytest

from oracle import numpy_ref as R

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from l3es import _native  # noqa: E402


@pytest.mark.parametrize("n,batch", [(16, 2), (32, 1)])
def test_long_runs_are_several_launches(n, batch):
    steps = 2500
    p = _native.Plan(dim=2, n=n, nu=5e-3, dt=1e-3, drag=0.1, kolm_k=2, kolm_amp=1.0, batch=batch)
    uh0 = np.stack([np.fft.rfftn(R.init_u_random2d(n, b, n / 4)[..., 0], axes=(1, 2)) for b in range(batch)])
    a = torch.from_numpy(np.ascontiguousarray(uh0, dtype=np.complex64)).cuda().reshape(p.spec_shape)
    b = a.clone()
    e_inj = torch.full((steps * batch,), np.nan, dtype=torch.float64, device="cuda")
    p.timing(True)
    p.step(a, steps, e_inj=e_inj)
    launches = sum(v[0] for v in p.kernel_stats().values())
    p.timing(False)
    assert 2 <= launches <= 25  # about 15 us a step: at 100 steps a launch their own cost is below 1 %
    for part in (1, 99, 1400, 1000):
        p.step(b, part)
    p.check()
    assert torch.equal(a, b)
    assert bool((e_inj == 0).all())
