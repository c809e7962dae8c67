"""The acoustic step's two column forms (one block per row segment of 32
columns; one thread per column above col_max_segments) bit for bit with the
FP32 oracle at the sizes where their index arithmetic can go wrong: row
segments of one column, one short of full, full and one over, the shortest
and the tallest column, the smallest domain accepted, odd widths (whose last pair of columns is half
inside), and a domain on each side of the size rule.  The FP64 column form
is compared between the two: a member alone takes one of them, in an ensemble
above the rule the other, and the fields agree bit for bit.

The same domains cover the level chunks of the other column kernels (one
level in the last chunk, chunks that a short member leaves empty) and the
row-segment forms of rk_step_prep and calc_coef_w on both sides of their
size rules.
"""
import pytest

from wrf_gb300 import cases
from wrf_gb300 import gpu as G

from _harness import OracleDomain
from test_gpu_parity import STATE_FIELDS, _bitwise_diffs
from wrf_gb300 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,kde", [(31, 9, 14), (32, 8, 15), (33, 10, 17), (64, 9, 33), (65, 8, 128),
                                       (12, 3011, 14), (33, 1510, 16), (31, 950, 14), (40, 1255, 15),
                                       (7, 7, 6), (33, 7, 7)])
def test_column_forms_bitwise(gpulib, nx, ny, kde):
    case = cases.small_case(nx=nx, ny=ny, kde=kde, n_scalar=1, seed=nx + kde)
    od = OracleDomain(case, "f32")
    ge = G.Domain(case)
    od.step(2)
    ge.step(2)
    ge.sync()
    bad = _bitwise_diffs(case, ge, od)
    assert not bad, "\n".join(bad)


@pytest.mark.parametrize("open_sides", [False, True])
def test_column_forms_bitwise_options(gpulib, open_sides):
    case = cases.small_case(nx=45, ny=20, kde=24, n_scalar=1, seed=3)
    if open_sides:
        case = cases.open_boundaries(case)
    c = case.desc.config
    c.damp_opt, c.dampcoef, c.zdamp, c.w_damping = 3, 0.2, 5000.0, 1
    od = OracleDomain(case, "f32")
    ge = G.Domain(case)
    od.step(2)
    ge.step(2)
    ge.sync()
    bad = _bitwise_diffs(case, ge, od)
    assert not bad, "\n".join(bad)


@pytest.mark.parametrize("kde", [14, 33, 128])
def test_fp64_column_forms_agree(gpulib, kde):
    a = cases.small_case(nx=33, ny=11, kde=kde, n_scalar=1, seed=kde)
    b = cases.small_case(nx=12, ny=1010, kde=kde, n_scalar=1, seed=kde + 1)
    alone = G.Domain(a, flags=G.FLAG_MIXED)
    both = G.Ensemble.from_cases([a, b], flags=G.FLAG_MIXED)
    for d in (alone, both):
        d.step(2)
        d.sync()
    for nm in STATE_FIELDS:
        fid = abi.FIELD_ID[nm]
        assert (alone.get(0, fid) == both.get(0, fid)).all(), nm


def test_level_chunks_of_uneven_members(gpulib):
    """One launch cuts every member's levels into the tallest member's chunks:
    members of 14, 43 and 128 levels, plain, each equal to its own run."""
    three = [cases.small_case(nx=20 + q, ny=9 + q, kde=kde, n_scalar=2, seed=q) for q, kde in enumerate((14, 43, 128))]
    ens = G.Ensemble.from_cases(three)
    ens.step(2)
    ens.sync()
    for q, case in enumerate(three):
        od = OracleDomain(case, "f32")
        od.step(2)
        bad = _bitwise_diffs(case, ens, od, member=q)
        assert not bad, "\n".join(bad)
