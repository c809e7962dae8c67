"""A host I/O step whose input of one field is the output buffer of another: a
step reads what the step before wrote there (wrfgpu_step_host), although a
passive scalar's download crosses the link during the next step."""
import numpy as np
import pytest

from wrf_gb300 import abi, cases
from wrf_gb300 import gpu as G

from test_host_io import _pinned

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [0, G.FLAG_NO_GRAPH], ids=["graph", "direct"])
def test_input_from_another_fields_output(gpulib, flags):
    """qv comes in from the buffer the last of eight passive scalars goes out to (fields of 4.5 MB, so that
    scalar's download is the last of eight on the link), three steps in one call: the scalars and qv bit for
    bit those of the set / step / get loop."""
    case = cases.small_case(nx=200, ny=260, kde=20, n_scalar=8, seed=12)
    ref, dut = G.Domain(case, flags), G.Domain(case, flags)
    sp = [abi.species_id(s) for s in range(9)]
    outs = [_pinned(dut.field_size(0, f)) for f in sp]
    qv_out, shared = outs[0], outs[8]
    shared[:] = np.asarray(ref.get(0, sp[8])).ravel()
    dut.bind_host_state(0, sp, [shared] + [None] * 8, outs)
    dut.step_host(3)
    x = np.array(ref.get(0, sp[8])).ravel()
    for _ in range(3):
        ref.set(0, sp[0], x)
        ref.step(1)
        ref.sync()
        x = np.array(ref.get(0, sp[8])).ravel()
    for f, b in zip(sp, outs):
        assert np.array_equal(b, np.asarray(ref.get(0, f)).ravel()), f
    dut.unbind_host_state()
