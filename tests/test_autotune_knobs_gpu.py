"""The autotuner leaves alone what its timed step does not reach (the right-hand side, irfftn
and the adjoint do), and does not read cache lines of other kernels."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from l3es import _native  # noqa: E402

KEYS = _native.Plan.SCHEDULE_KEYS


@pytest.mark.parametrize("dim,n,reached", [
    (2, 16, ""), (2, 64, ""), (2, 128, ""), (2, 256, "line_pair"), (2, 512, ""), (3, 32, ""), (3, 64, ""),
    (3, 128, "y_radix8 line_pair band_bulk")])
@pytest.mark.parametrize("value", [0, 1])
def test_unreached_knobs_stay(dim, n, reached, value):
    for _ in range(4):
        p = _native.Plan(dim=dim, n=n, nu=1e-3, dt=1e-4)
        p.set_schedule({k: value for k in KEYS})
        got = p.autotune("")
        assert all(got[k] == value for k in KEYS if k not in reached.split()), got


def test_lines_of_other_kernels_are_not_read(tmp_path):
    """A line as builds wrote it before the key named the kernels."""
    cap = torch.cuda.get_device_capability()
    name = torch.cuda.get_device_name().replace(" ", "_")
    cache = tmp_path / "sched.txt"
    p = _native.Plan(dim=2, n=64, nu=1e-3, dt=1e-4)
    start = p.schedule
    other = " ".join(str(1 - start[k]) for k in KEYS)
    line = f"{name}|sm{cap[0]}{cap[1]}|d2|n64|b1|f{p.step_form} {other}\n"
    cache.write_text(line)
    assert p.autotune(str(cache)) == start
    lines = cache.read_text().splitlines(keepends=True)
    assert lines[0] == line and len(lines) == 2


def test_routes_do_not_share_a_line(tmp_path):
    """Plans of one size and form whose steps run different kernels (a Kolmogorov wavenumber
    beyond the stored band, the integrating factor) have lines of their own."""
    cache = str(tmp_path / "sched.txt")
    for kw in ({}, dict(kolm_k=26, kolm_amp=1.0), dict(scheme="integrating_factor")):
        _native.Plan(dim=2, n=64, nu=1e-3, dt=1e-4, **kw).autotune(cache)
    assert len(open(cache).read().splitlines()) == 2  # the last two take the same kernels
