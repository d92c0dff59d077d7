"""The memory pool behind the operator calls: memory is given back, calls on several streams and threads stay apart.

Exact comparisons: the same call on the same inputs gives the same bits whatever ran before or beside it.
"""
import ctypes as C
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _setup(dims=(8, 8, 8, 8), ls=8, n=2):
    import torch
    import cps_public_b200 as cb
    from cps_public_b200 import fields
    cb.init(0)
    g = cb.Gauge(fields.random_gauge(dims, 0.2, 81), dims)
    op = cb.DiracOp(g, "dwf", mass=0.1, ls=ls)
    b = torch.from_numpy(np.stack([fields.random_source(op.n // 24, 82 + q) for q in range(n)])).cuda()
    torch.cuda.synchronize()
    return cb, op, b


def _mdagm(op, b, prec, stream=None):
    import torch
    from cps_public_b200 import _lib
    lib = _lib.load()
    out = torch.empty_like(b)
    torch.cuda.synchronize()
    _lib.check(lib.cpsb_mdagm_multi_dev(op.gauge.h, C.byref(op.p), prec, b.shape[0], C.c_void_p(out.data_ptr()),
                                        C.c_void_p(b.data_ptr()), None, stream), "cpsb_mdagm_multi_dev")
    return out.cpu().numpy()


def test_memory_is_given_back():
    cb, op, b = _setup((16, 16, 16, 16), 16, 1)
    _mdagm(op, b, cb.F64)
    free0, _ = cb.mem_info()
    for _ in range(3):
        _mdagm(op, b, cb.F64)
    free1, _ = cb.mem_info()
    assert abs(free1 - free0) < 64 << 20, (free0, free1)  # a vector here is 100 MB


def test_threads_and_streams_stay_apart():
    import torch
    cb, op, b = _setup()
    want = {p: _mdagm(op, b, p) for p in (cb.F64, cb.F32, cb.F16)}
    bad = []

    def work(prec):
        st = torch.cuda.Stream()
        for _ in range(20):
            if not np.array_equal(_mdagm(op, b, prec, st.cuda_stream), want[prec]):
                bad.append(prec)

    th = [threading.Thread(target=work, args=(p,)) for p in want for _ in range(2)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not bad


def test_refused_call_leaves_the_pool_usable():
    cb, op, b = _setup()
    want = _mdagm(op, b, cb.F64)
    bad = cb.DiracOp(op.gauge, "mobius", mass=0.1, ls=5)  # no kernels for this Ls: refused after the call has begun
    with pytest.raises(cb.CpsbError):
        bad.MatPc(np.zeros(bad.n))
    assert np.array_equal(_mdagm(op, b, cb.F64), want)


def _small(cb):
    """Loads every kernel of the large calls below."""
    cb, op, b = _setup((8, 8, 8, 8), 16, 8)
    _mdagm(op, b, cb.F64)


def test_memory_of_a_large_call_is_given_back():
    """Free memory as reported right after a call of 3.2 GB of vectors is what it was before the call."""
    import torch
    cb, op, b = _setup((16, 16, 16, 16), 16, 8)
    _small(cb)
    out = torch.empty_like(b)
    del out  # stays with torch, for the result of the call
    free0, _ = cb.mem_info()
    _mdagm(op, b, cb.F64)
    free1, _ = cb.mem_info()
    assert free0 - free1 < 64 << 20, (free0, free1)


LAST_GAUGE = """
import torch
from tests.test_gpu_call_pool import _mdagm, _setup, _small
cb, op, b = _setup((16, 16, 16, 16), 16, 8)
_small(cb)
out = torch.empty_like(b)
del out  # stays with torch, for the result of the call
cb.mem_info()
free0 = torch.cuda.mem_get_info()[0]
_mdagm(op, b, cb.F64)
kept = free0 - torch.cuda.mem_get_info()[0]
op.gauge.free()
freed = torch.cuda.mem_get_info()[0]
assert kept > 2 << 30, kept         # what the pool keeps between calls
assert free0 - freed < 64 << 20, (free0, freed)
"""


def test_last_gauge_gives_the_pool_back():
    """A process of its own: no other gauge field may be resident."""
    import pathlib
    import subprocess
    import sys
    root = pathlib.Path(__file__).resolve().parents[1]
    r = subprocess.run([sys.executable, "-c", LAST_GAUGE], cwd=root, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]


def test_request_loop_beside_refused_calls():
    """Requests, each of which records its own graph, while another thread's calls are refused for lack of memory."""
    import torch
    from cps_public_b200 import _lib, fields
    cb, opb, b = _setup((16, 16, 16, 16), 16, 8)
    g = cb.Gauge(fields.random_gauge((4, 4, 4, 4), 0.2, 83), (4, 4, 4, 4))
    op = cb.DiracOp(g, "dwf", mass=0.1, ls=4)
    src = fields.random_source(op.n // 24, 84)
    lib, out = _lib.load(), torch.empty_like(b)
    free, _ = cb.mem_info()
    ballast = torch.empty(free - (1 << 30), dtype=torch.uint8, device="cuda")
    stop, codes = threading.Event(), []

    def refused():
        while not stop.is_set():
            codes.append(lib.cpsb_mdagm_multi_dev(opb.gauge.h, C.byref(opb.p), cb.F64, b.shape[0],
                                                  C.c_void_p(out.data_ptr()), C.c_void_p(b.data_ptr()), None, None))

    th = threading.Thread(target=refused)
    srv = cb.Server(slots=3, hbm_bytes=400 << 20)
    th.start()
    try:
        first = {}
        for _ in range(15):
            ids = [(p, srv.submit(op, [src], stop_rsd=1e-8, precision=p)) for p in (cb.F32, cb.F16, cb.F32)]
            for p, i in ids:
                xs = srv.wait(i)[0]
                assert np.array_equal(first.setdefault(p, xs[0]), xs[0])
    finally:
        stop.set()
        th.join()
        srv.close()
        del ballast
        torch.cuda.empty_cache()
    assert set(codes) == {-3}  # out of memory, nothing else
