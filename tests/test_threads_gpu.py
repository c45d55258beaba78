"""Calls of several host threads, each on its own plan and stream, on grids whose kernels take
different amounts of shared memory: none fails, and the results are those of calls in turn."""
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from l3es import _native  # noqa: E402


def test_exact_sums_of_several_grids_at_once():
    calls = []
    for c in (8, 64, 16, 32):
        rng = np.random.default_rng(c)
        p = _native.InterpPlan(dim=3, ckp_n=c, n_fine=0, np_max=64)
        p.set_field(torch.from_numpy(rng.standard_normal((3, c, c, c)).astype(np.float32)).cuda())
        r = torch.from_numpy(rng.uniform(0.0, 2 * np.pi, (5, 3))).cuda()
        out, ref = torch.empty_like(r), torch.empty_like(r)
        p.interp(r, ref, backend="dft")
        grid = torch.empty((3, c, c, c), device="cuda")
        grid_ref = torch.empty_like(grid)
        p.particles_to_grid(r, ref, grid_ref)
        calls.append((p, r, out, ref, grid, grid_ref))
    torch.cuda.synchronize()
    errors = []

    def run(p, r, out, ref, grid, grid_ref):
        try:
            s = torch.cuda.Stream()
            for _ in range(400):
                p.interp(r, out, backend="dft", stream=s)
                p.particles_to_grid(r, ref, grid, stream=s)
            s.synchronize()
        except Exception as e:  # reported by the test's thread
            errors.append(e)

    threads = [threading.Thread(target=run, args=a) for a in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
    for _, _, out, ref, grid, grid_ref in calls:
        assert torch.equal(out, ref) and torch.equal(grid, grid_ref)
