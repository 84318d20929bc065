"""GPU: what plan options still vary -- slab depths, the cap on resident derivative CTAs, chunks --
changes no bit of a right-hand side, an RK4 stage or the constraints, on rows that end in
tiles of every width; the default plan stays pinned to the oracle."""
import numpy as np
import pytest

import sympygr_b200 as sg
from oracle import pyoracle as po
from sympygr_b200 import workloads as wl

pytestmark = pytest.mark.gpu

# rows of 7 to 36 interior points: last tiles of 3 to 16 columns, odd and even numbers of tiles
SIZES = [(nx, 13 + nx % 5, 13 + nx % 3) for nx in range(13, 43)]
FLAGS = (0x00, 0x3F, 0x12, 0x00, 0x29)


def _batch():
    rng = np.random.default_rng(5)
    blocks, off = [], 0
    for k, sz in enumerate(SIZES):
        h = rng.uniform(0.02, 0.06, 3)
        pmin = rng.uniform(-0.9, 0.4, 3)
        off += int(rng.integers(0, 9))
        blocks.append(wl.Block(off, sz, FLAGS[k % 5], tuple(map(float, pmin)),
                               tuple(float(pmin[a] + (sz[a] - 1) * h[a]) for a in range(3))))
        off += sz[0] * sz[1] * sz[2]
    u = np.zeros((24, off))
    for b in blocks:
        x, y, z = wl.coords(b)
        u[:, b.offset:b.offset + b.npad] = po.fake_initial_data(x, y, z).reshape(24, -1)
    return u, blocks


def _eval(ctx, ud, blocks, precision, advective, **kw):
    import torch

    plan = sg.Plan(ctx, blocks, precision, advective=advective, **kw)
    prm = sg.Params.make(ko_sigma=0.2, precision=precision)
    rhs, con, step = torch.zeros_like(ud), torch.zeros((4, ud.shape[1]), dtype=ud.dtype, device="cuda"), ud.clone()
    plan.rhs_device(list(rhs), list(ud), prm)
    plan.constraints_device(list(ud), list(con))
    rk = sg.RK4(plan)
    rk.init(list(step))
    rk.step(list(step), 1e-3, prm)
    torch.cuda.synchronize()
    rk.close()
    plan.close()
    return rhs, con, step


@pytest.mark.parametrize("precision", [sg.FP64, sg.MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("advective", [False, True], ids=["centred", "upwind"])
def test_options_change_no_bit(ctx, oracle_lib, precision, advective):
    import torch

    u, blocks = _batch()
    ud = torch.from_numpy(u).cuda()
    ref = _eval(ctx, ud, blocks, precision, advective)
    if precision == sg.FP64:
        oracle, got = po.oracle_rhs_adv if advective else po.oracle_rhs, ref[0].cpu().numpy()
        for b in blocks:
            mx, _ = po.rel_errors(po.interior(got, b), po.interior(oracle(u, b, po.params(ko_sigma=0.2)), b))
            assert mx.max() < 1e-12, (b, mx.max())
    for kw in ({"slab_depth": 3}, {"slab_depth": 5, "block_slab_depth": [k % 8 for k in range(len(blocks))]},
               {"deriv_ctas_per_sm": 1}, {"chunk_points": 3000}):
        for name, a, b in zip(("right-hand side", "constraints", "RK4 step"), ref, _eval(ctx, ud, blocks, precision, advective, **kw)):
            assert torch.equal(a, b), (kw, name)
