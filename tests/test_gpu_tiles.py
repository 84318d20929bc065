"""GPU: the derivative stage at the edges of its tiles and slabs.

Extents just below, at and above a tile's 16 x 8 columns (with remainders of one and two
points, which the cut moves into the tile before), slabs down to three planes, odd block
offsets (rows that start off a 16-byte boundary) and flagged faces on each of them."""
import numpy as np
import pytest

import sympygr_b200 as sg
from oracle import pyoracle as po
from sympygr_b200 import workloads as wl

pytestmark = pytest.mark.gpu

SIZES = [(13, 13, 13), (21, 14, 16), (22, 15, 13), (23, 23, 14), (24, 16, 19), (25, 31, 15), (38, 22, 13), (39, 14, 17)]


def _block(sz, flags, offset):
    pmin, h = (-0.37, 0.11, -0.23), (0.031, 0.027, 0.043)
    blk = wl.Block(offset, sz, flags, pmin, tuple(pmin[a] + (sz[a] - 1) * h[a] for a in range(3)))
    x, y, z = wl.coords(blk)
    u = np.zeros((24, offset + blk.npad))
    u[:, offset:] = po.fake_initial_data(x, y, z).reshape(24, -1)
    return u, blk


@pytest.mark.parametrize("sz", SIZES)
def test_derivatives_equal_the_oracle_bit_for_bit(ctx, oracle_lib, sz):
    for flags in (0x00, 0x3F, 0x15, 0x2A, 0x30):
        u, blk = _block(sz, flags, 0)
        rhs = np.zeros_like(u)
        ctx.bssnrhs(list(rhs), list(u), 0, blk.pmin, blk.pmax, blk.sz, flags, sg.Params.make(ko_sigma=0.2))
        assert np.array_equal(ctx.debug_block_scratch(blk.ninterior), po.oracle_slots(u, blk)), hex(flags)


@pytest.mark.parametrize("precision", [sg.FP64, sg.MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("advective", [False, True], ids=["centred", "upwind"])
def test_slab_cuts_do_not_change_the_result(ctx, precision, advective):
    import torch

    parts, blocks, off = [], [], 0
    for k, sz in enumerate(SIZES):
        u, blk = _block(sz, (0x00, 0x3F, 0x26, 0x11)[k % 4], 1 + k % 3)
        parts.append(u)
        blocks.append(wl.Block(off + blk.offset, blk.sz, blk.bflag, blk.pmin, blk.pmax))
        off += u.shape[1]
    ud = torch.from_numpy(np.concatenate(parts, 1)).cuda()
    prm = sg.Params.make(ko_sigma=0.2, precision=precision)
    out = []
    for depth in (0, 1, 4, 7, 66):
        plan = sg.Plan(ctx, blocks, precision, slab_depth=depth, advective=advective)
        rd = torch.zeros_like(ud)
        plan.rhs_device(list(rd), list(ud), prm)
        torch.cuda.synchronize()
        plan.close()
        out.append(rd)
    for depth, rd in zip((1, 4, 7, 66), out[1:]):
        assert torch.equal(rd, out[0]), depth
    ref = po.oracle_rhs_adv if advective else po.oracle_rhs
    if precision == sg.FP64:
        got = out[0].cpu().numpy()
        u = ud.cpu().numpy()
        for b in blocks:
            mx, _ = po.rel_errors(po.interior(got, b), po.interior(ref(u, b, po.params(ko_sigma=0.2)), b))
            assert mx.max() < 1e-12, (b, mx.max())
