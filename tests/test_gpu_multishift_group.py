"""MInvCG with its shifts updated per group of iterations: groups cut short, one shift, limits inside a group.

The reference is one InvCg on the shifted operator's residual equation, formed here: every converged shift must satisfy
|b - (A + s) x| <= 4 stop |b| in FP64 (the reported residual is the iterated one; at 1e-8 the drift between the two
is far below the factor).  batch = 1, 3, 4, 5 makes groups of 1, 3, 4, and 4 + 1 iterations; the same arithmetic in
the same order on every element, so they must agree bit for bit when the iteration count is the same.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHIFTS = np.array([1e-3, 5e-3, 0.02, 0.3, 2.0])


def _op(action, ls):
    import cps_public_b200 as cb
    from cps_public_b200 import fields
    cb.init(0)
    dims = (4, 4, 4, 8)
    g = cb.Gauge(fields.random_gauge(dims, 0.2, 91), dims)
    op = cb.DiracOp(g, action, mass=0.1, ls=ls)
    return cb, op, [fields.random_source(op.n // 24, 92 + q) for q in range(2)]


def _solve(cb, op, srcs, shifts, prec, batch, ms_type, max_iter=2000, stop=1e-8):
    import torch
    from cps_public_b200 import _lib
    lib = _lib.load()
    nv, ns = len(srcs), len(shifts)
    nsol = 1 if ms_type == cb.SINGLE else ns
    b = torch.from_numpy(np.stack(srcs)).cuda()
    x = torch.zeros(nv, nsol, op.n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    xp = (C.c_void_p * (nv * nsol))(*[x[q, s].data_ptr() for q in range(nv) for s in range(nsol)])
    rsd = np.full((nv, ns), stop)
    al = 1.0 + np.arange(ns)
    arg = cb.CgArg(stop, max_iter, prec, 0.1, batch)
    res = (cb.SolveResult * nv)()
    rc = lib.cpsb_minvcg_multi_dev(op.gauge.h, C.byref(op.p), C.byref(arg), nv, xp, C.c_void_p(b.data_ptr()),
                                   _lib.ptr(np.ascontiguousarray(shifts)), ns, _lib.ptr(rsd), ms_type, _lib.ptr(al),
                                   res, None)
    assert rc >= 0
    return x.cpu().numpy(), [r.iters for r in res], rc


@pytest.mark.parametrize("action,ls", [("wilson", 1), ("dwf", 5), ("mobius", 4)])
def test_groups_agree_and_solve(action, ls):
    cb, op, srcs = _op(action, ls)
    x0 = None
    for batch in (1, 3, 4, 5):
        x, it, rc = _solve(cb, op, srcs, SHIFTS, cb.F64, batch, cb.MULTI)
        assert rc == 0
        if x0 is None:
            x0, it0 = x, it
            for q, b in enumerate(srcs):
                for s, sh in enumerate(SHIFTS):
                    ax, _ = op.MatPcDagMatPc(x[q, s])
                    assert np.linalg.norm(b - ax - sh * x[q, s]) <= 4e-8 * np.linalg.norm(b), (q, s)
        assert it == it0 and np.array_equal(x, x0), batch
    single, _, _ = _solve(cb, op, srcs, SHIFTS, cb.F64, 4, cb.SINGLE)
    want = np.einsum("s,qsn->qn", 1.0 + np.arange(len(SHIFTS)), x0)
    # the weighted sum in another order: rounding of a few hundred updates per element
    assert np.linalg.norm(single[:, 0] - want) <= 1e-12 * np.linalg.norm(want)
    for batch in (1, 5):
        again, _, _ = _solve(cb, op, srcs, SHIFTS, cb.F64, batch, cb.SINGLE)
        assert np.array_equal(again, single), batch


def test_one_shift_and_limit_inside_a_group():
    cb, op, srcs = _op("dwf", 4)
    one, _, rc = _solve(cb, op, srcs, SHIFTS[:1], cb.F64, 4, cb.MULTI)
    assert rc == 0
    for q, b in enumerate(srcs):
        ax, _ = op.MatPcDagMatPc(one[q, 0])
        assert np.linalg.norm(b - ax - SHIFTS[0] * one[q, 0]) <= 4e-8 * np.linalg.norm(b)
    for limit in (1, 2, 6):  # the limit ends the solve in the middle of a group
        xs = [_solve(cb, op, srcs, SHIFTS, cb.F64, batch, cb.MULTI, max_iter=limit) for batch in (1, 4)]
        assert xs[0][2] == xs[1][2] == 1 and xs[0][1] == xs[1][1]
        assert np.array_equal(xs[0][0], xs[1][0]), limit


@pytest.mark.parametrize("action,ls", [("wilson", 1), ("dwf", 5), ("mobius", 4)])
def test_fp32_groups_agree(action, ls):
    """FP32 Krylov vectors (16-byte chunks of four reals): groups of every length do the operations of one pass per
    iteration, so the refinement starts from the same solutions and neither it nor the result may differ."""
    cb, op, srcs = _op(action, ls)
    x0, it0, rc = _solve(cb, op, srcs, SHIFTS, cb.F32, 1, cb.MULTI, stop=1e-10)
    assert rc == 0
    for batch in (3, 4, 5):
        x, it, rc = _solve(cb, op, srcs, SHIFTS, cb.F32, batch, cb.MULTI, stop=1e-10)
        assert rc == 0 and it == it0 and np.array_equal(x, x0), batch
