"""The energy sums of the field statistics and of the spectrum keep FP64's bits: terms 2^-26
and 2^-52 of the largest, in one thread's share, whose sum FP64 holds and 48 bits do not."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from l3es import _native  # noqa: E402

TERMS = [1.0, 2.0**-13] + [2.0**-26] * 6  # amplitudes of eight terms
SUM = 1.0 + 2.0**-26 + 6 * 2.0**-52       # of their squares


@pytest.mark.parametrize("dim", [2, 3])
def test_field_statistics(dim):
    n = 16
    p = _native.Plan(dim=dim, n=n, nu=1e-2, dt=1e-3)
    u = torch.zeros(p.phys_shape, dtype=torch.float32, device="cuda")
    u[0].view(-1)[:8] = torch.tensor(TERMS)
    out = torch.empty(4, dtype=torch.float64, device="cuda")
    p.field_stats(u, out)
    assert float(out[3]) == 0.5 * SUM / n**dim  # powers of two beside the sum


def test_spectrum():
    n, kh = 16, 1
    p = _native.Plan(dim=3, n=n, nu=1e-2, dt=1e-3)
    uh = torch.zeros(p.spec_shape, dtype=torch.complex64, device="cuda")
    rows = [(2, 1), (14, 1), (2, 15), (14, 15), (1, 2), (15, 2), (1, 14), (15, 14)]
    for (x, y), v in zip(rows, TERMS):
        uh[0, x, y, kh] = v
    ek = torch.empty(n, dtype=torch.float64, device="cuda")
    p.energy_spectrum(uh, ek)
    k = np.fft.fftfreq(n, 1.0 / n)
    kz = np.arange(n // 2 + 1)
    shell = (np.sqrt(k[:, None, None] ** 2 + k[None, :, None] ** 2 + kz**2) + 0.5).astype(int)
    count = ((shell == 2) * np.where((kz == 0) | (kz == n // 2), 1.0, 2.0)).sum()
    ref = 2.0 * SUM / n**6 * 4.0 * np.pi * 4.0 / (count + np.finfo(float).eps)
    # the product and the quotient round twice on each side; the terms lost at 48 bits are 12 units
    assert abs(float(ek[2]) - ref) <= 4 * 2.0**-53 * ref
