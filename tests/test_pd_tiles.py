"""The routine-level advect_scalar_pd (one tiled kernel, level chunks) bit for
bit with the FP32 oracle where its tiles can go wrong: domains of one partial
tile, exactly one tile, one column or row over, the shortest column and one
cut into many level chunks, periodic and open on all sides; and, on device
arrays whose rows are neither 16-byte aligned nor a multiple of 16 bytes,
equal to the host-array entry point (test_zz_no_alloc's calls).
"""
import numpy as np
import pytest

from wrf_gb300 import abi, cases
from wrf_gb300 import gpu as G

from _harness import OracleDomain, interior, max_abs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,kde,open_sides", [(12, 8, 14, False), (31, 9, 15, False), (32, 8, 60, False),
                                                  (33, 17, 33, True), (65, 24, 128, False), (40, 25, 21, True)])
def test_routine_pd_bitwise(gpulib, nx, ny, kde, open_sides):
    case = cases.small_case(nx=nx, ny=ny, kde=kde, n_scalar=1, seed=nx + kde)
    if open_sides:
        case = cases.open_boundaries(case)
    od = OracleDomain(case, "f32")
    ge = G.Domain(case)
    od.step(1)
    ge.step(1)
    ge.sync()
    for sp in (0, 1):
        od.run("advect_scalar_pd", 3, 0, sp)
        ge.run_routine("advect_scalar_pd", 3, 0, sp)
        ge.sync()
        fid = abi.FIELD_ID["advect_tend"]
        a, b = interior(case, fid, ge.get(0, fid)), interior(case, fid, od.get(fid))
        assert float(np.max(np.abs(b))) > 0.0
        assert max_abs(a, b) == 0.0
