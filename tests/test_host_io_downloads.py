"""The downloads of a host I/O call's last step: fields stored to host memory
by the pack kernel (up to 2 MB) and staged ones, the positive-definite
transport in one, two and three groups of pairs with each group's species
downloaded before the swap, and a call of several steps; the buffers equal
the fields read one by one afterwards, and the state a run without bound
buffers, bit for bit."""
import numpy as np
import pytest

from wrf_gb300 import abi, cases
from wrf_gb300 import gpu as G

from test_host_io import _fids, _pinned

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,kde,nsc,open_sides,nsteps", [
    (20, 12, 14, 0, False, 1), (33, 20, 14, 4, True, 2), (200, 260, 14, 10, False, 1), (200, 260, 14, 9, True, 1),
    (320, 420, 14, 10, False, 3)])
def test_last_step_downloads(gpulib, nx, ny, kde, nsc, open_sides, nsteps):
    case = cases.small_case(nx=nx, ny=ny, kde=kde, n_scalar=nsc, seed=nx)
    if open_sides:
        case = cases.open_boundaries(case)
    ref = G.Domain(case)
    dut = G.Domain(case)
    fids = _fids(case)
    outs = [_pinned(dut.field_size(0, f)) for f in fids]
    dut.bind_host_state(0, fids, [None] * len(fids), outs)
    for n in (nsteps, 1):
        dut.step_host(n)
        ref.step(n)
        ref.sync()
        for f, b in zip(fids, outs):
            assert np.array_equal(b, np.asarray(ref.get(0, f)).ravel()), (n, f)
            assert np.array_equal(b, np.asarray(dut.get(0, f)).ravel()), (n, f)
    dut.unbind_host_state()
