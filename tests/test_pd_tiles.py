"""The routine-level advect_scalar_pd (one tiled kernel, level chunks) bit for
bit with the FP32 oracle where its tiles can go wrong: domains of one partial
tile, exactly one tile, one column or row over, the shortest column and one
cut into many level chunks, periodic and open on all sides; and, on device
arrays whose rows are neither 16-byte aligned nor a multiple of 16 bytes,
equal to the host-array entry point (test_zz_no_alloc's calls).
"""
import ctypes as C

import numpy as np
import pytest

from wrf_gb300 import abi, cases
from wrf_gb300 import gpu as G

from _harness import OracleDomain, interior, max_abs
from test_fortran_abi import _fid, _scalars, _state
from test_zz_no_alloc import NAMES, _Args, _dims, _routine_call

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

def _device_call(lib, case, dev, tend, scal, stream):
    """wrfgpu_advect_scalar_pd_noalloc's argument list on `stream`: (function, arguments, what they point to)."""
    a = _Args()
    a.ptr(dev["qv"].data_ptr()); a.ptr(dev["qv_old"].data_ptr()); a.ptr(tend.data_ptr())
    for nm in ("ru_m", "rv_m", "ww_m", "c1h", "c2h", "muts", "mub", "mu_1"):
        a.ptr(dev[nm].data_ptr())
    a.cfg(case.desc.config)
    for nm in ("msftx", "msfty", "fnm", "fnp"):
        a.ptr(dev[nm].data_ptr())
    a.f32(scal["rdx"]); a.f32(scal["rdy"]); a.ptr(dev["rdnw"].data_ptr()); a.f32(scal["dtrk"])
    for d in _dims(case):
        a.i32(d)
    a.args.append(C.c_void_p(stream))
    fn = lib.wrfgpu_advect_scalar_pd_noalloc
    fn.restype = C.c_int
    fn.argtypes = [C.c_void_p] * len(a.args)
    return fn, a.args, a


def test_device_calls_of_two_threads(gpulib):
    """Two host threads, each on its own stream, over columns of 14 and of 128 levels: the kernel's shared
    memory depends on the height, and neither thread's calls may be refused or changed by the other's.  Every
    call accumulates onto the thread's tendency, whose end state equals the same calls made alone."""
    import threading

    torch = pytest.importorskip("torch")
    ncall = 2000
    jobs = []
    for kde in (14, 128):
        case = cases.small_case(nx=16, ny=12, kde=kde, n_scalar=0, seed=kde)
        od = _state(case)
        dev = {nm: torch.from_numpy(np.ascontiguousarray(od.get(_fid(nm)), dtype=np.float32)).cuda() for nm in NAMES}
        n = np.asarray(od.get(abi.FIELD_ID["advect_tend"])).size
        tends = [torch.zeros(n, device="cuda") for _ in range(2)]
        stream = torch.cuda.Stream()
        calls = [_device_call(gpulib, case, dev, t, _scalars(case, 3, 1), stream.cuda_stream) for t in tends]
        jobs.append((dev, tends, calls))
    torch.cuda.synchronize()

    def many(call):
        fn, args, _ = call
        return [rc for rc in (fn(*args) for _ in range(ncall)) if rc != 0]

    for _, _, calls in jobs:  # alone, one thread after the other
        assert many(calls[0]) == []
    refused = {}
    ready = threading.Barrier(2)

    def work(q):
        ready.wait()
        refused[q] = many(jobs[q][2][1])

    threads = [threading.Thread(target=work, args=(q,)) for q in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert refused == {0: [], 1: []}
    for _, tends, _ in jobs:
        assert float(tends[0].abs().max()) > 0.0
        assert torch.equal(tends[0], tends[1])

@pytest.mark.parametrize("nx,ny,kde,open_sides", [(8, 8, 6, False), (13, 8, 14, False), (32, 8, 60, False),
                                                  (33, 17, 33, True), (65, 24, 128, False), (40, 25, 21, True)])
def test_device_arrays_bitwise(gpulib, nx, ny, kde, open_sides):
    """One partial tile, exactly one, a column or row over, three tile columns, the shortest and the tallest
    column, on a stream of its own, every array one float past a 16-byte boundary: the first call, onto zeros,
    gives the oracle's tendency, and the second, onto the first's, what the host-array entry point gives."""
    torch = pytest.importorskip("torch")
    case = cases.small_case(nx=nx, ny=ny, kde=kde, n_scalar=0, seed=nx + kde)
    if open_sides:
        case = cases.open_boundaries(case)
    od = _state(case)
    host = {nm: np.ascontiguousarray(od.get(_fid(nm)), dtype=np.float32) for nm in NAMES}
    scal = _scalars(case, 3, 1)
    fid = abi.FIELD_ID["advect_tend"]

    def unaligned(a):
        base = torch.zeros(a.size + 4, device="cuda")
        out = base[1:1 + a.size]
        out.copy_(torch.from_numpy(a))
        assert out.data_ptr() % 16 == 4
        return out

    dev = {nm: unaligned(host[nm]) for nm in NAMES}
    tend = unaligned(np.zeros(np.asarray(od.get(fid)).size, np.float32))
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    fn, args, _ = _device_call(gpulib, case, dev, tend, scal, stream.cuda_stream)
    assert fn(*args) == 0
    stream.synchronize()
    first = tend.cpu().numpy()
    assert fn(*args) == 0
    stream.synchronize()
    second = tend.cpu().numpy()

    od.run("advect_scalar_pd", 3, 0, 0)
    b = interior(case, fid, od.get(fid))
    assert float(np.max(np.abs(b))) > 0.0
    assert max_abs(interior(case, fid, first), b) == 0.0
    ref = first.copy()
    assert _routine_call(gpulib, case, host, ref, scal) == 0
    assert np.array_equal(interior(case, fid, second), interior(case, fid, ref))
    assert not np.array_equal(first, second)
    for nm in NAMES:  # the inputs stay as they were
        assert np.array_equal(dev[nm].cpu().numpy(), host[nm])


def test_device_call_under_capture(gpulib):
    """The call is one kernel of a captured graph: each replay accumulates once more."""
    torch = pytest.importorskip("torch")
    case = cases.small_case(nx=33, ny=9, kde=20, n_scalar=0, seed=5)
    od = _state(case)
    dev = {nm: torch.from_numpy(np.ascontiguousarray(od.get(_fid(nm)), dtype=np.float32)).cuda() for nm in NAMES}
    n = np.asarray(od.get(abi.FIELD_ID["advect_tend"])).size
    direct, captured = torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
    scal = _scalars(case, 3, 1)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        stream = torch.cuda.current_stream().cuda_stream
        fn, args, keep = _device_call(gpulib, case, dev, captured, scal, stream)
        rc = fn(*args)
    assert rc == 0
    fn, args, keep2 = _device_call(gpulib, case, dev, direct, scal, 0)
    for _ in range(3):
        graph.replay()
        assert fn(*args) == 0
    torch.cuda.synchronize()
    assert float(direct.abs().max()) > 0.0
    assert torch.equal(direct, captured)
