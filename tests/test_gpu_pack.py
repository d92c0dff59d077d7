"""Host (CPS) order <-> device layout through the operator boundary, at the edges of the packing tiles.

DslashPrec packs its input, hops and unpacks the result.  A tile holds floor(128 / C) sites of C slices, so the
lattices and Ls here give tiles that end inside the lattice, columns of 1 to 32 entries (odd ones among them), two
classes of unequal height (odd DWF Ls) and one class (Wilson, Mobius).  The reference is the C oracle; FP64 to the
rounding of 8 neighbours' 3x3 products (1e-13), FP32 to 2e-6, 16-bit storage to 5e-4, the bounds of the launch-shape
test.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = {0: 1e-13, 1: 2e-6, 2: 5e-4}


@pytest.mark.parametrize("dims,action,ls", [((4, 6, 4, 6), "wilson", 1), ((2, 2, 2, 4), "wilson", 1),
                                            ((4, 4, 6, 4), "dwf", 2), ((4, 6, 4, 6), "dwf", 5),
                                            ((4, 6, 6, 4), "dwf", 11), ((2, 4, 2, 6), "dwf", 64),
                                            ((4, 4, 4, 6), "mobius", 12), ((4, 2, 4, 6), "mobius", 32)])
def test_pack_tiles(dims, action, ls):
    import cps_public_b200 as cb
    from cps_public_b200 import fields
    from oracle import oracle
    cb.init(0)
    u = fields.random_gauge(dims, 0.3, 71)
    g = cb.Gauge(u, dims)
    op = cb.DiracOp(g, action, mass=0.1, ls=ls)
    ref = oracle.Op(action, dims, u, ls=ls, mass=0.1)
    src = fields.random_source(int(np.prod(dims)) // 2 * ls, 72)
    for cb_, dag in ((1, 0), (0, 1)):
        want = ref.dslash(src, cb_, dag)
        for prec in (0, 1, 2):
            got = op.DslashPrec(src, cb_, dag, prec)
            err = np.linalg.norm(got - want) / np.linalg.norm(want)
            assert err < TOL[prec], (cb_, dag, prec, err)
