"""Mobius CG with the residual update inside the last hop + M5 kernel, against the separate update.

CPSB_M5_FUSE=0 runs the hops, the M5 passes and the CG update as kernels of their own.  Both solve to the same FP64
true residual 1e-10, so on these 4^3x6 lattices (condition below 1e3) the solutions agree to 1e-7 relative at the
worst; FP64 iteration counts differ by rounding at most (within one).  Ls at both ends of the range and with tiles
that end inside a block; a zero source among three right-hand sides; the shifted update through the refinement of a
reduced-precision multishift solve.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = (4, 4, 4, 6)


def _op(ls, fused, monkeypatch):
    import cps_public_b200 as cb
    from cps_public_b200 import fields
    monkeypatch.setenv("CPSB_M5_FUSE", "1" if fused else "0")
    cb.init(0)
    g = cb.Gauge(fields.random_gauge(DIMS, 0.2, 101), DIMS, bc_t=1)
    return cb, cb.DiracOp(g, "mobius", mass=0.1, ls=ls)


@pytest.mark.parametrize("ls", [4, 12, 20, 32])
@pytest.mark.parametrize("prec", [0, 1, 2])
def test_fused_update_matches_separate(ls, prec, monkeypatch):
    from cps_public_b200 import fields
    out = []
    for fused in (True, False):
        cb, op = _op(ls, fused, monkeypatch)
        srcs = [fields.random_source(op.n // 24, 102), np.zeros(op.n), fields.random_source(op.n // 24, 103)]
        xs, rs = op.InvCgMulti(srcs, stop_rsd=1e-10, precision=prec)
        assert all(r.status == 0 and r.true_rsd <= 1e-10 for r in rs)
        assert not xs[1].any()
        out.append((xs, [r.iters for r in rs]))
    for q in (0, 2):
        a, b = out[0][0][q], out[1][0][q]
        assert np.linalg.norm(a - b) <= 1e-7 * np.linalg.norm(b)
        if prec == 0:
            assert abs(out[0][1][q] - out[1][1][q]) <= 1


def test_shifted_update(monkeypatch):
    from cps_public_b200 import fields
    cb, op = _op(8, True, monkeypatch)
    src = fields.random_source(op.n // 24, 104)
    shifts = [1e-3, 0.05, 1.0]
    xs, r, rs = op.MInvCG(src, shifts, [1e-10] * 3, precision=cb.F32)
    assert r.status == 0 and max(rs) <= 1e-10
    for s, x in zip(shifts, xs):
        ax, _ = op.MatPcDagMatPc(x)
        assert np.linalg.norm(src - ax - s * x) <= 1.01e-10 * np.linalg.norm(src)
