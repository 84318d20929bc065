"""GPU: the allocation-free entry point at the edges of its cuts: rows and columns that leave one
to four points beyond whole tiles, slabs of three and four planes, tiles whose scratch starts off a
32-point boundary, with and without flagged faces.  Its result is that of the plans.

Named so that pytest collects it last, like the other tests of this entry point."""
import pytest

import sympygr_b200 as sg
from test_zz_no_alloc import TOL64, TOL_MIXED, _check, _elongated, _pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [(sg.FP64, TOL64), (sg.MIXED, TOL_MIXED)], ids=["fp64", "mixed"])
@pytest.mark.parametrize("sz", [(23, 15, 13), (24, 16, 14), (25, 23, 17), (39, 24, 19), (15, 33, 31), (71, 13, 28)])
def test_noalloc_at_the_cuts(ctx, sz, precision, tol):
    for flags in (0x00, 0x3F, 0x26):
        u, blk = _elongated(sz, flags)
        a, b = _pair(ctx, u, blk, 0.3, precision)
        _check(a, b, blk, tol)
