"""SPH neighbour lists that the density pass leaves for the acceleration pass: particles with
more neighbours than a lane's list holds (a clustered half) beside a lattice, against a plan
too large to keep lists (it searches in both passes), to the bit; and positions on the box's
faces and outside it, where the quotient by the box side is an integer or large."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from l3es import _native  # noqa: E402

L = 2 * np.pi
# np_max above which a plan keeps no lists (1 GiB of 8 lanes x (32 + 1 or 12 + 1) words)
LARGE = {3: 1_100_000, 2: 2_700_000}


def _positions(dim, n, seed):
    rng = np.random.default_rng(seed)
    m = n**dim
    r = rng.uniform(0.0, L, (m, dim))
    r[: m // 2] = 0.7 + rng.uniform(0.0, L / 4, (m // 2, dim))  # a crowd
    r[-1], r[-2], r[-3] = 0.0, L, -3 * L
    r[-4], r[-5], r[-6] = np.nextafter(L, 0.0), -1e-17, 41.25 * L
    return torch.from_numpy(r).cuda(), torch.from_numpy(rng.standard_normal((m, dim))).cuda()


@pytest.mark.parametrize("dim,n", [(3, 9), (3, 13), (2, 9), (2, 40)])
def test_kept_lists_match_the_search(dim, n):
    r, u = _positions(dim, n, n)
    outs = []
    for np_max in (r.shape[0], LARGE[dim]):
        p = _native.SphPlan(dim, n, L, np_max=np_max)
        o = [torch.empty_like(r) for _ in range(6)]
        p.relax_acceleration(r, o[0], 4.0)
        p.forces(r, u, o[1], o[2], o[3], 4.0)
        p.relax_velocity(r, u, o[4], 2e-3, 2.0, 4.0, r_out=o[5])
        outs.append(o)
        del p
    for a, b in zip(*outs):
        assert torch.equal(a, b)
    assert bool(torch.isfinite(outs[0][0]).all())
    moved = outs[0][5].cpu().numpy()
    ref = np.mod(r.cpu().numpy() + 2e-3 * outs[0][4].cpu().numpy(), L)
    gap = np.abs(moved - ref)
    # wrapped into [0, L); three roundings of numbers up to 42 L beside the reference's own
    assert moved.min() >= 0.0 and moved.max() < L
    assert np.minimum(gap, L - gap).max() <= 4 * 42 * L * 2.0**-52
