"""Every launch of a step is allowed its shared memory, on every device and for
every height.  A kernel's allowance of more than 48 KB belongs to the device
it was set on, so a process that steps domains on two devices has to set it on
both; and no launch may lower what another thread's taller launch relies on.
The step's launches are checked on the CPU against a runtime that runs no
kernel and keeps the allowances (tests/native/fake_cudart.c)."""
import os
import shutil
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

CHILD = """
import ctypes as C, sys
from wrf_gb300 import cases
from wrf_gb300 import gpu as G
fake = C.CDLL(sys.argv[1])
nx, ny, flags, damp = (int(a) for a in sys.argv[2:])
for device, kde in ((0, 128), (0, 14), (1, 14), (1, 128), (0, 60)):
    fake.fake_set_device(device)
    case = cases.small_case(nx=nx, ny=ny, kde=kde, n_scalar=1, seed=3)
    if damp:
        case.desc.config.damp_opt, case.desc.config.zdamp, case.desc.config.dampcoef = 3, 5000.0, 0.2
    dom = G.Domain(case, flags=flags | G.FLAG_NO_GRAPH)
    before, refused = fake.fake_launches(), fake.fake_refused()
    rc = dom.L.wrfgpu_step(dom.h, 1)
    assert fake.fake_launches() - before > 60
    assert (rc, fake.fake_refused() - refused) == (0, 0), (device, kde)
    dom.run_routine("advect_scalar_pd", 3, 0, 0)
    assert fake.fake_refused() == refused, (device, kde)
    dom.close()
assert fake.fake_lowered() == 0
print("allowed")
"""


# the row-segment kernels (plain, mixed, damped), then the marches of a domain of more segments
@pytest.mark.skipif(shutil.which("gcc") is None, reason="gcc not available")
@pytest.mark.parametrize("nx,ny,flags,damp", [(12, 10, 0, 0), (12, 10, 1, 1), (8, 1010, 1, 0), (8, 3010, 0, 1)])
def test_step_on_two_devices(tmp_path, nx, ny, flags, damp):
    if not os.path.exists(os.path.join(ROOT, "wrf_gb300", "libwrfgpu.so")):
        import __graft_entry__ as g
        g.build()
    fake = str(tmp_path / "fake_cudart.so")
    subprocess.run(["gcc", "-O1", "-shared", "-fPIC", "-o", fake, os.path.join(HERE, "native", "fake_cudart.c")],
                   check=True)
    r = subprocess.run([sys.executable, "-c", CHILD, fake, str(nx), str(ny), str(flags), str(damp)], cwd=ROOT,
                       env=dict(os.environ, LD_PRELOAD=fake), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.strip().endswith("allowed")
