"""Handles on the GPU: calls from several host threads, and the cost of creating one."""
import ctypes as C
import os
import shutil
import statistics
import subprocess
import threading
import time

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def _dev():
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    return torch.device("cuda:0")


@pytest.fixture(scope="module")
def loops(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    out = str(tmp_path_factory.mktemp("loops") / "libloops.so")
    subprocess.check_call([gxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-o", out,
                           os.path.join(HERE, "cpp", "call_loop.cpp")])
    return C.CDLL(out)


def _vp(t):
    return C.c_void_p(t.data_ptr())


def _tables(nsp, nrc, ntb, nt, tmp):
    from openhurricane_b200 import synth
    from openhurricane_b200.mechanism import compile_mechanism
    m = synth.make_mechanism(nsp, nrc, ntb, nt, seed=5 + nsp)
    return compile_mechanism(*synth.write_chemkin(m, str(tmp / f"m{nsp}")))


def _cells(t, n, dev):
    from openhurricane_b200 import synth
    c = synth.dirichlet_cells(t.nsp, n, seed=n, T_range=(800.0, 2800.0), alpha=0.3)
    d = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)
    return d(c.T), d(c.p), d(synth.mixture_density(t.W, c)), d(c.Y)


def _all_at_once(jobs):
    """(loop function, its arguments before the stream, outputs) each in a thread and a stream
    of its own; every call must be accepted and leave what it leaves alone."""
    streams = [torch.cuda.Stream() for _ in jobs]
    rcs, start = [None] * len(jobs), threading.Barrier(len(jobs))

    def work(k, loop, fn, reps, args):
        start.wait()
        rcs[k] = loop(fn, reps, *args, C.c_void_p(streams[k].cuda_stream))

    alone = []
    for k, (loop, fn, reps, args, outs) in enumerate(jobs):
        assert loop(fn, 1, *args, C.c_void_p(streams[k].cuda_stream)) == 0
        torch.cuda.synchronize()
        alone.append([o.clone() for o in outs])
    ts = [threading.Thread(target=work, args=(k, *j[:4])) for k, j in enumerate(jobs)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    torch.cuda.synchronize()
    assert rcs == [0] * len(jobs), rcs
    for (_, _, _, _, outs), was in zip(jobs, alone):
        assert all(torch.equal(a, b) for a, b in zip(outs, was))


def test_properties_of_many_and_few_cells_in_two_threads(loops, large):
    """One handle; the two calls take different amounts of shared memory."""
    from openhurricane_b200 import _capi
    from openhurricane_b200.chemistry import Mechanism
    dev, t = _dev(), large["tables"]
    m, lib, jobs, held = Mechanism(t), _capi.load(), [], []
    fn = C.cast(lib.hc_properties, C.c_void_p)
    for n, reps in ((20000, 5000), (64, 20000)):
        T, p, rho, Y = _cells(t, n, dev)
        out = [torch.empty_like(Y)] + [torch.empty_like(T) for _ in range(3)] + [torch.empty_like(Y)]
        held.append((T, p, Y))
        args = [m.handle, C.c_int64(n)] + [_vp(a) for a in (T, p, Y, *out)]
        jobs.append((loops.loop_properties, fn, reps, args, out))
    _all_at_once(jobs)
    m.close()


def test_jacobians_of_two_mechanisms_in_two_threads(loops, tmp_path):
    """Two mechanisms of one kernel size whose tables differ in size."""
    from openhurricane_b200 import _capi
    from openhurricane_b200.chemistry import Mechanism
    dev, lib, jobs, held = _dev(), _capi.load(), [], []
    fn = C.cast(lib.hc_rhs_jacobian, C.c_void_p)
    for shape in ((17, 60, 10, 4), (31, 120, 20, 6)):
        t = _tables(*shape, tmp_path)
        m, n = Mechanism(t), 50
        T, p, rho, Y = _cells(t, n, dev)
        c = (rho[None] * Y / torch.tensor(t.W, device=dev)[:, None]).contiguous()
        out = [torch.empty((n, t.nsp + 1), dtype=torch.float64, device=dev),
               torch.empty((n, t.nsp + 1, t.nsp + 1), dtype=torch.float64, device=dev)]
        held.append((m, T, p, c))
        jobs.append((loops.loop_jacobian, fn, 20000,
                     [m.handle, C.c_int64(n)] + [_vp(a) for a in (c, T, p, *out)], out))
    _all_at_once(jobs)
    for h in held:
        h[0].close()


@pytest.mark.parametrize("name,pairs", [("small", 30), ("large", 45)])
def test_creating_a_handle_takes_few_allocations(name, pairs, request):
    """The device tables come in one allocation and one copy. The bar is the time of that many
    allocations and copies; with one for each table a handle took over 60 and the packing
    of the tables (the large mechanism's is half of what it takes now)."""
    rt = pytest.importorskip("cuda.bindings.runtime")
    from openhurricane_b200 import _capi
    _dev()
    tables = request.getfixturevalue(name)["tables"]
    lib = _capi.load()
    desc = _capi.DescArrays(tables)
    part = np.zeros(4096, np.uint8)
    torch.cuda.synchronize()

    def create():
        h = C.c_void_p()
        assert lib.hc_mech_create(C.byref(desc.desc), C.byref(h)) == 0
        lib.hc_mech_destroy(h)

    def allocate():
        held = []
        for _ in range(pairs):
            err, q = rt.cudaMalloc(65536)
            assert int(err) == 0
            held.append(q)
            rt.cudaMemcpy(q, part.ctypes.data, part.nbytes, rt.cudaMemcpyKind.cudaMemcpyHostToDevice)
        for q in held:
            rt.cudaFree(q)

    def median(f):
        ts = []
        for _ in range(25):
            t0 = time.perf_counter()
            f()
            ts.append(time.perf_counter() - t0)
        return statistics.median(ts[5:])

    took, bar = median(create), median(allocate)
    assert took <= bar, (took, bar)
