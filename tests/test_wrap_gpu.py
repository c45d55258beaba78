"""The periodic wrap at the edges of its branch (a position inside the box stays as it is):
the box's faces and their neighbours, signed zeros, subnormals, many periods, infinities and
NaN, and boxes the branch must not take (negative, infinite). Against floor division in FP64."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from l3es import _native  # noqa: E402


@pytest.mark.parametrize("box", [2 * np.pi, 1.0, 1.9999999999999998, 3e-5, -2.0, np.inf])
def test_wrap_edges(box):
    b = box if np.isfinite(box) else 1.0
    x = np.array([0.0, -0.0, 5e-324, -5e-324, b, np.nextafter(b, 0), np.nextafter(b, 2 * b), -b, 2 * b, 0.5 * b,
                  -0.25 * b, 1e6 * b, -1e6 * b, np.nextafter(2 * b, 0), np.inf, -np.inf, np.nan])
    r = torch.from_numpy(x).cuda()
    out = _native.shift(r, torch.zeros_like(r), scale=1.0, box=box).cpu().numpy()
    with np.errstate(all="ignore"):
        q = np.floor(x / box)
        ref = x - box * q
        ref = np.where(ref >= box, ref - box, ref)
        # the product's rounding (contracted on the device)
        tol = np.abs(box * q) * 2.0**-52
    bad = ~np.isfinite(ref)
    assert np.array_equal(np.isnan(out), np.isnan(ref))
    assert np.all(np.abs(out[~bad] - ref[~bad]) <= tol[~bad])
    inside = (x >= 0) & (x < box) & np.isfinite(x) & np.isfinite(box)
    assert np.array_equal(out[inside], x[inside])
