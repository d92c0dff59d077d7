"""MInvCG with FP32 Krylov vectors where device memory is short.

The updates of the upper shifts go faster with three more residuals per source, which the call may take only where they
are not needed: a first call builds its refinement solver after the Krylov phase, and a call that has room for one
residual runs with one.  The rest of the device is held by one torch tensor meanwhile.  Both calls do the same operations
on every element as an unhindered one, so the solutions agree bit for bit.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS, LS, NV, NS = (16, 16, 16, 16), 8, 4, 2
MB = 1 << 20


class _Case:
    def __init__(self):
        import torch
        import cps_public_b200 as cb
        from cps_public_b200 import fields
        self.cb, self.torch = cb, torch
        cb.init(0)
        self.u = fields.random_gauge(DIMS, 0.2, 111)
        self.n = int(np.prod(DIMS)) // 2 * LS
        gen = torch.Generator(device="cuda").manual_seed(112)
        self.b = torch.randn(NV, self.n * 24, dtype=torch.float64, device="cuda", generator=gen)
        self.x = torch.empty(NV, NS, self.n * 24, dtype=torch.float64, device="cuda")
        # device bytes: the Krylov phase with one residual (source, solutions, two temporaries of the operator, A p,
        # p_s, psi_s, r) and the refinement solver (x, b, r and two temporaries of one source in FP64; r, p, A p, x and
        # two temporaries in FP32)
        self.f32, f64 = NV * self.n * 96, NV * self.n * 192
        self.krylov = f64 * (1 + NS) + self.f32 * (2 + 1 + 2 * NS + 1)
        self.solver = 3 * f64 + 2 * f64 // NV + 6 * self.f32
        self.slack = 100 * MB  # links, reduction slots, the pool's granularity

    def gauge(self):
        return self.cb.Gauge(self.u, DIMS)

    def solve(self, g):
        from cps_public_b200 import _lib
        lib = _lib.load()
        op = self.cb.DiracOp(g, "dwf", mass=0.1, ls=LS)
        self.x.zero_()
        self.torch.cuda.synchronize()
        shifts, rsd, al = np.array([1e-3, 0.1]), np.full((NV, NS), 1e-9), np.ones(NS)
        xp = (C.c_void_p * (NV * NS))(*[self.x[q, s].data_ptr() for q in range(NV) for s in range(NS)])
        arg = self.cb.CgArg(1e-9, 3000, self.cb.F32, 0.1, 0)
        res = (self.cb.SolveResult * NV)()
        _lib.check(lib.cpsb_minvcg_multi_dev(g.h, C.byref(op.p), C.byref(arg), NV, xp, C.c_void_p(self.b.data_ptr()),
                                             _lib.ptr(shifts), NS, _lib.ptr(rsd), self.cb.MULTI, _lib.ptr(al), res,
                                             None), "cpsb_minvcg_multi_dev")
        return [r.iters for r in res]

    def leave(self, n):
        """A tensor that leaves n bytes of the device free."""
        free, _ = self.cb.mem_info()
        assert free > n
        return self.torch.empty(free - n, dtype=self.torch.uint8, device="cuda")


def test_first_call_has_room_for_its_refinement():
    """Room for the Krylov phase, the refinement solver and half of the three spare residuals."""
    c = _Case()
    g = c.gauge()
    iters = c.solve(g)
    want = c.x.clone()
    g.free()  # and its refinement solver
    g = c.gauge()
    ballast = c.leave(c.krylov + c.solver + 3 * c.f32 // 2 + c.slack)
    try:
        assert c.solve(g) == iters
    finally:
        del ballast
        c.torch.cuda.empty_cache()
    assert c.torch.equal(c.x, want)
    g.free()


def test_later_call_runs_with_one_residual():
    """The refinement solver is there; room for the Krylov phase and half of the spare residuals."""
    c = _Case()
    g = c.gauge()
    iters = c.solve(g)
    want = c.x.clone()
    ballast = c.leave(c.krylov + 3 * c.f32 // 2 + c.slack)
    try:
        assert c.solve(g) == iters
    finally:
        del ballast
        c.torch.cuda.empty_cache()
    assert c.torch.equal(c.x, want)
    g.free()
