"""The forward diffusion by columns and the edge strips of all species at once,
bit for bit with the FP32 oracle where their index arithmetic can go wrong:
level chunks of one level and chunks whose first vertical flux is formed
below them, tiles one column wide, each subset of the terms (horizontal and
vertical alone, sixth order alone, both, next to open boundaries one without
the other), and the limiter factors of the narrowest domain whose strips do
not overlap, with one side open, the other, and both.
"""
import pytest

from wrf_gb300 import cases
from wrf_gb300 import gpu as G

from _harness import OracleDomain
from test_gpu_parity import _bitwise_diffs

pytestmark = pytest.mark.gpu


def _compare(case):
    od = OracleDomain(case, "f32")
    ge = G.Domain(case)
    od.step(2)
    ge.step(2)
    ge.sync()
    bad = _bitwise_diffs(case, ge, od, old_too=False)
    assert not bad, "\n".join(bad)


@pytest.mark.parametrize("diff,sixth", [(1, 0), (0, 2), (1, 2)])
@pytest.mark.parametrize("nx,ny,kde,open_sides", [(33, 9, 14, False), (32, 17, 33, False), (12, 12, 66, True),
                                                  (45, 20, 24, True)])
def test_forward_diffusion_bitwise(gpulib, nx, ny, kde, open_sides, diff, sixth):
    case = cases.small_case(nx=nx, ny=ny, kde=kde, n_scalar=2, seed=nx + kde)
    if open_sides:
        case = cases.open_boundaries(case)
    c = case.desc.config
    if diff:
        c.diff_opt, c.km_opt, c.khdif, c.kvdif = 1, 1, 75.0, 8.0
    if sixth:
        c.diff_6th_opt, c.diff_6th_slopeopt, c.diff_6th_factor, c.diff_6th_thresh = sixth, 1, 0.12, 0.10
    c.damp_opt, c.dampcoef, c.zdamp = 2, 0.01, 8000.0
    _compare(case)


@pytest.mark.parametrize("nx,ny,sides", [(11, 9, "x"), (9, 11, "y"), (11, 11, "xy"), (12, 40, "xy"), (70, 13, "xy")])
def test_strips_of_all_species_bitwise(gpulib, nx, ny, sides):
    case = cases.small_case(nx=nx, ny=ny, kde=15, n_scalar=5, seed=nx + ny)
    case = cases.open_boundaries(case, x="x" in sides, y="y" in sides)
    _compare(case)
