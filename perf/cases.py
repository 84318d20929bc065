"""Performance cases of the BSSN right-hand side: what its users call, over the sizes they call it with.

A relativity code reaches this library in four ways, and every case below is one of them:

* block by block on host arrays, through the drop-in for the reference's ``bssnrhs``;
* block by block on device arrays, through the allocation-free entry point;
* as a plan over an octree's block list (right-hand sides, constraints), on device or host arrays;
* as RK4 steps of such a plan, replayed from a CUDA graph.

Each case is a dict of plain values; ``prepare`` turns it into a state, ``run`` makes one pass.
The fields are those of an evolution under way: the two-puncture data of the benchmark with a
smooth perturbation of every variable (amplitude 1e-3, as the sine block's), so no right-hand
side vanishes.  ``exact`` restates the whole evaluation in plain torch, in 64 bits.
"""
import math

import numpy as np
import torch

import sympygr_b200 as sg
from sympygr_b200 import capi, workloads as wl
from sympygr_b200.workloads import Block

NUM_VARS = 24
SIGMA = 0.1          # Kreiss-Oliger strength of the cases
OCTREE = (13, 21, 37, 69, 135)          # padded block sizes of the octree batch
OCTREE_COUNTS = (1800, 750, 300, 120, 30)  # and how many of each a full batch has


def listed():
    return [
        # One octree leaf through the drop-in: the smallest call there is (60 % of an octree's
        # blocks have this size); launches, copies and host work count, not arithmetic.
        {"name": "dropin_13_fp64", "kind": "dropin", "nx": 13, "ny": 13, "nz": 13, "flags": 0x15, "mixed": False},
        # A large block through the drop-in, as a host code's block loop calls it.
        {"name": "dropin_69_mixed", "kind": "dropin", "nx": 69, "ny": 69, "nz": 69, "flags": 0, "mixed": True},
        # The allocation-free entry point at its largest block, inside another framework's step.
        {"name": "noalloc_38_fp64", "kind": "noalloc", "nx": 38, "ny": 38, "nz": 38, "flags": 0, "mixed": False},
        # One small block resident on the device: a refinement level with a single box.
        {"name": "block_21_mixed", "kind": "plan", "layout": "single", "nx": 21, "ny": 21, "nz": 21, "flags": 0x3F,
         "mixed": True, "upwind": False},
        # The single-puncture box with Sommerfeld values on all six faces.
        {"name": "block_134_fp64", "kind": "plan", "layout": "single", "nx": 134, "ny": 134, "nz": 134, "flags": 0x3F,
         "mixed": False, "upwind": False},
        # A quarter of the benchmark's octree batch, in both precisions: one stage of a production run.
        {"name": "octree_fp64", "kind": "plan", "layout": "octree", "scale": 0.25, "mixed": False, "upwind": False},
        {"name": "octree_mixed", "kind": "plan", "layout": "octree", "scale": 0.25, "mixed": True, "upwind": False},
        # Blocks that are not cubes, of odd and even extents, at any offset, some with flagged faces.
        {"name": "ragged_fp64", "kind": "plan", "layout": "ragged", "blocks": 48, "lo": 13, "hi": 75, "mixed": False,
         "upwind": False},
        # The opt-in upwind advection.
        {"name": "upwind_mixed", "kind": "plan", "layout": "octree", "scale": 0.125, "mixed": True, "upwind": True},
        # The constraint monitor between steps: fields and block norms.
        {"name": "constraints_fp64", "kind": "constraints", "layout": "octree", "scale": 0.125, "mixed": False},
        # One RK4 step of an evolution on a tiled cube, Sommerfeld on its outer faces, from a graph.
        {"name": "rk4_mixed", "kind": "rk4", "layout": "tiled", "tiles": 4, "n": 37, "mixed": True},
        # The batch from page-locked host arrays, copied in and out in pieces that overlap the kernels.
        {"name": "host_mixed", "kind": "host", "layout": "octree", "scale": 0.0625, "mixed": True},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def scale(lo, hi):
        return round(math.exp(rng.uniform(math.log(lo), math.log(hi))), 4)

    kind = rng.choice(["dropin", "noalloc", "single", "single", "octree", "octree", "octree", "ragged", "ragged", "upwind",
                       "constraints", "rk4", "rk4", "host"])
    mixed = rng.random() < 0.5
    flags = rng.choice([0, 0, 0x3F, rng.randrange(1, 64)])
    if kind == "dropin":
        return {"kind": "dropin", "nx": size(13, 90), "ny": size(13, 90), "nz": size(13, 90), "flags": flags, "mixed": mixed}
    if kind == "noalloc":
        return {"kind": "noalloc", "nx": size(13, 38), "ny": size(13, 38), "nz": size(13, 38), "flags": flags, "mixed": mixed}
    if kind == "single":
        return {"kind": "plan", "layout": "single", "nx": size(13, 150), "ny": size(13, 150), "nz": size(13, 150),
                "flags": flags, "mixed": mixed, "upwind": rng.random() < 0.25}
    if kind == "ragged":
        lo = size(13, 30)
        return {"kind": "plan", "layout": "ragged", "blocks": size(2, 48), "lo": lo, "hi": lo + size(4, 45),
                "mixed": mixed, "upwind": rng.random() < 0.25}
    if kind == "rk4":
        return {"kind": "rk4", "layout": "tiled", "tiles": rng.randrange(2, 5), "n": size(13, 45), "mixed": mixed}
    if kind == "constraints":
        return {"kind": "constraints", "layout": "octree", "scale": scale(1 / 64, 1 / 8), "mixed": mixed}
    if kind == "host":
        return {"kind": "host", "layout": "octree", "scale": scale(1 / 64, 1 / 16), "mixed": mixed}
    if kind == "upwind":
        return {"kind": "plan", "layout": "octree", "scale": scale(1 / 64, 1 / 8), "mixed": mixed, "upwind": True}
    return {"kind": "plan", "layout": "octree", "scale": scale(1 / 64, 1 / 4), "mixed": mixed, "upwind": False}


# ---------------------------------------------------------------------------- block lists

def _single(n, flags):
    """One block whose interior spans [-8, 8] along its longest axis, with one spacing."""
    h = 16.0 / (max(n) - 7)
    pmin = tuple(-0.5 * (n[a] - 1) * h for a in range(3))
    return Block(0, tuple(n), flags, pmin, tuple(pmin[a] + (n[a] - 1) * h for a in range(3)))


def _layout(case, seed):
    """(blocks, elements per variable) of a case."""
    if "nx" in case:
        n = (case["nx"], case["ny"], case["nz"])
        return [_single(n, case["flags"])], n[0] * n[1] * n[2]
    if case["layout"] == "octree":
        counts = tuple(max(1, int(round(c * case["scale"]))) for c in OCTREE_COUNTS)
        return wl.batch_blocks(OCTREE, counts, seed)
    if case["layout"] == "tiled":
        return wl.tiled_domain_blocks(case["tiles"], case["n"], 8.0)
    # the shapes of a ragged list belong to the case, its place and its flags to the seed
    shapes = np.random.default_rng(case["blocks"] * 1000003 + case["lo"] * 1009 + case["hi"])
    rng = np.random.default_rng(seed)
    blocks, off = [], 0
    for _ in range(case["blocks"]):
        n = tuple(int(x) for x in shapes.integers(case["lo"], case["hi"] + 1, 3))
        gap = int(shapes.integers(0, 40))
        h = 1.0 / (max(n) - 7)
        lo = rng.uniform(-6.0, 5.0, 3)
        flag = int(rng.integers(1, 64)) if rng.uniform() < 0.25 else 0
        pmin = tuple(float(lo[a] - 3 * h) for a in range(3))
        blocks.append(Block(off, n, flag, pmin, tuple(pmin[a] + (n[a] - 1) * h for a in range(3))))
        off += n[0] * n[1] * n[2] + gap
    return blocks, off


def _coordinates(blocks, total, device):
    """x, y, z of every padded point (0 in the gaps between blocks)."""
    xyz = torch.zeros((3, total), dtype=torch.float64, device=device)
    by_shape = {}
    for b in blocks:
        by_shape.setdefault(tuple(b.sz), []).append(b)
    for (nx, ny, nz), group in by_shape.items():
        step = max(1, (1 << 25) // (nx * ny * nz))
        for s in range(0, len(group), step):
            part = group[s:s + step]
            at = torch.tensor([b.offset for b in part], device=device)[:, None] + torch.arange(nx * ny * nz, device=device)
            for a, n in enumerate((nx, ny, nz)):
                h = torch.tensor([b.h[a] for b in part], dtype=torch.float64, device=device)[:, None]
                p = torch.tensor([b.pmin[a] for b in part], dtype=torch.float64, device=device)[:, None]
                line = p + h * torch.arange(n, dtype=torch.float64, device=device)
                shape = [len(part), 1, 1, 1]
                shape[3 - a] = n
                xyz[a].index_copy_(0, at.reshape(-1), line.reshape(shape).expand(len(part), nz, ny, nx).reshape(-1))
    return xyz


def _fields(blocks, total, seed, device):
    """[24, total]: two-puncture data plus two sine modes of amplitude up to 1e-3 in every variable."""
    rng = np.random.default_rng(seed)
    xyz = _coordinates(blocks, total, device)
    u = torch.zeros((NUM_VARS, total), dtype=torch.float64, device=device)
    psi = torch.ones(total, dtype=torch.float64, device=device)
    for px in (-4.0, 4.0):
        psi += 0.25 / torch.sqrt((xyz[0] - px) ** 2 + xyz[1] ** 2 + xyz[2] ** 2 + 1e-4)
    u[wl.U_CHI] = psi ** -4
    u[wl.U_ALPHA] = psi ** -2
    for v in (wl.U_SYMGT0, wl.U_SYMGT3, wl.U_SYMGT5):
        u[v] = 1.0
    for v in range(NUM_VARS):
        for _ in range(2):
            k = rng.uniform(0.5, 3.0, 3)
            wave = xyz[0] * k[0]
            wave.add_(xyz[1], alpha=k[1]).add_(xyz[2], alpha=k[2]).add_(rng.uniform(0.0, 2 * math.pi))
            u[v].add_(wave.sin_(), alpha=rng.uniform(-1e-3, 1e-3))
    # the conformal factor and the lapse stay positive next to a puncture
    u[wl.U_CHI].clamp_(min=1e-4)
    u[wl.U_ALPHA].clamp_(min=1e-2)
    return u


# ---------------------------------------------------------------------------- the library

_CONTEXT = None


def _context():
    """A program's one context: it is made once and every plan and call shares it."""
    global _CONTEXT
    if _CONTEXT is None:
        _CONTEXT = sg.Context(0)
    return _CONTEXT


def _params(case):
    return sg.Params.make(ko_sigma=SIGMA, precision=sg.MIXED if case["mixed"] else sg.FP64,
                          ghost_policy=sg.GHOSTS_ZERO if case["kind"] == "host" else sg.GHOSTS_PRESERVE)


def prepare(case, seed):
    blocks, total = _layout(case, seed)
    u = _fields(blocks, total, seed, "cuda")
    kind, precision = case["kind"], sg.MIXED if case["mixed"] else sg.FP64
    state = {"kind": kind, "blocks": blocks, "total": total, "prm": _params(case)}
    if kind == "dropin":
        state["u"] = u.cpu().numpy()
        state["rhs"] = np.zeros_like(state["u"])
    elif kind == "host":
        state["u"] = torch.empty((NUM_VARS, total), dtype=torch.float64, pin_memory=True).copy_(u)
        state["rhs"] = torch.zeros((NUM_VARS, total), dtype=torch.float64).pin_memory()
        state["plan"] = sg.Plan(_context(), blocks, precision, chunk_points=1 << 21)
    else:
        state["u"] = u
        if kind == "noalloc":
            state["rhs"] = torch.zeros_like(u)
        elif kind == "plan":
            state["rhs"] = torch.zeros_like(u)
            state["plan"] = sg.Plan(_context(), blocks, precision, advective=case["upwind"])
        elif kind == "constraints":
            state["con"] = torch.zeros((4, total), dtype=torch.float64, device="cuda")
            state["norms"] = torch.zeros((len(blocks), 8), dtype=torch.float64, device="cuda")
            state["plan"] = sg.Plan(_context(), blocks, precision)
        else:
            state["plan"] = sg.Plan(_context(), blocks, precision)
            state["rk"] = sg.RK4(state["plan"])
            state["rk"].init(list(u))
            state["rk"].capture(list(u), _dt(blocks), state["prm"], 1)
    return state


def _dt(blocks):
    return 0.25 * min(min(b.h) for b in blocks)


def run(state):
    kind, u, prm = state["kind"], state["u"], state["prm"]
    if kind == "dropin":
        b = state["blocks"][0]
        _context().bssnrhs(list(state["rhs"]), list(u), b.offset, b.pmin, b.pmax, b.sz, b.bflag, prm)
        return state["rhs"]
    if kind == "noalloc":
        capi.rhs_noalloc(list(state["rhs"]), list(u), state["blocks"][0], prm,
                         torch.cuda.current_stream().cuda_stream)
        return state["rhs"]
    if kind == "plan":
        state["plan"].rhs_device(list(state["rhs"]), list(u), prm)
        return state["rhs"]
    if kind == "host":
        state["plan"].rhs_host([r.numpy() for r in state["rhs"]], [f.numpy() for f in u], state["total"], prm)
        return state["rhs"]
    if kind == "constraints":
        state["plan"].constraints_device(list(u), list(state["con"]), state["norms"])
        return {"con": state["con"], "norms": state["norms"]}
    state["rk"].launch()
    return u


def work(case):
    """The state read over the padded blocks, the outputs written at interior points; the operations of
    the stencils (12 per first derivative, 14 per second and per dissipation row) and of the algebra."""
    blocks, _ = _layout(case, 0)
    padded = sum(b.npad for b in blocks)
    inside = sum(b.ninterior for b in blocks)
    if case["kind"] == "constraints":
        return {"bytes": 8 * (17 * padded + 4 * inside), "flops": 2935 * inside}
    point = 6973
    if case.get("upwind"):
        point += 72 * 10
    if case["kind"] == "rk4":
        point = 4 * (point + 4 * NUM_VARS)
    return {"bytes": 8 * NUM_VARS * (padded + inside), "flops": point * inside}


# ---------------------------------------------------------------------------- 64-bit restatement

# One-dimensional operators: {offset: weight}.  The closure rows next to a flagged face count their
# offsets from the first (last) interior point and replace the centred row at the three points there.
_D1 = ({-3: -1, -2: 9, -1: -45, 1: 45, 2: -9, 3: 1},
       [{0: -25, 1: 48, 2: -36, 3: 16, 4: -3}, {0: -3, 1: -10, 2: 18, 3: -6, 4: 1}, {0: 1, 1: -8, 3: 8, 4: -1}])
_D2 = ({-3: 2, -2: -27, -1: 270, 0: -490, 1: 270, 2: -27, 3: 2},
       [{0: 35, 1: -104, 2: 114, 3: -56, 4: 11}, {0: 11, 1: -20, 2: 6, 3: 4, 4: -1},
        {0: -1, 1: 16, 2: -30, 3: 16, 4: -1}])
_KO = ({-3: -1, -2: 6, -1: -15, 0: 20, 1: -15, 2: 6, 3: -1},
       [{0: -1, 1: 3, 2: -3, 3: 1}, {0: 3, 1: -10, 2: 12, 3: -6, 4: 1}, {0: -3, 1: 12, 2: -19, 3: 15, 4: -6, 5: 1}])


def _take(f, dim, lo, hi):
    return f.narrow(dim, lo, hi - lo)


def _row(f, dim, at, count, row, sign=1):
    """sum of weight * f over `count` points from index `at` along `dim`."""
    acc = None
    for off, w in row.items():
        t = _take(f, dim, at + sign * off, at + sign * off + count)
        acc = t * float(w) if acc is None else acc.add_(t, alpha=float(w))
    return acc


def _operator(f, axis, h, flags, op, centre, closure, odd):
    """An operator along `axis` (0 = x) at that axis' interior points; other points are 0."""
    dim, n = 3 - axis, f.shape[3 - axis]
    out = torch.zeros_like(f)
    _take(out, dim, 3, n - 3).copy_(_row(f, dim, 3, n - 6, op[0]) * centre)
    if flags >> (2 * axis) & 1:
        for r in range(3):
            _take(out, dim, 3 + r, 4 + r).copy_(_row(f, dim, 3, 1, op[1][r]) * closure[r])
    if flags >> (2 * axis + 1) & 1:
        for r in range(3):
            _take(out, dim, n - 4 - r, n - 3 - r).copy_(_row(f, dim, n - 4, 1, op[1][r], -1) * (closure[r] * odd))
    return out


def _d1(f, axis, h, flags):
    return _operator(f, axis, h, flags, _D1, 1 / (60 * h), [1 / (12 * h)] * 3, -1.0)


def _d2(f, axis, h, flags):
    return _operator(f, axis, h, flags, _D2, 1 / (180 * h * h), [1 / (12 * h * h)] * 3, 1.0)


def _ko(f, axis, h, flags):
    return _operator(f, axis, h, flags, _KO, -1 / (64 * h), [48 / (64 * s * h) for s in (59.0, 43.0, 49.0)], 1.0)


_UP = [{-1: -3, 0: -10, 1: 18, 2: -6, 3: 1}, {-3: -1, -2: 6, -1: -18, 0: 10, 1: 3}]  # /12h: beta > 0, otherwise
_HALF = [{0: -3, 1: 4, 2: -1}, {-1: -1, 1: 1}, {-2: 1, -1: -4, 0: 3}]                # /2h: forward, centred, backward


def _upwind(f, axis, h, flags, beta):
    dim, n = 3 - axis, f.shape[3 - axis]
    out = torch.zeros_like(f)

    def put(at, count, pos, neg):
        scale = {0: 1 / (12 * h), 1: 1 / (12 * h), 2: 1 / (2 * h), 3: 1 / (2 * h), 4: 1 / (2 * h)}
        rows = _UP + _HALF
        b = _take(beta, dim, at, at + count)
        _take(out, dim, at, at + count).copy_(torch.where(b > 0, _row(f, dim, at, count, rows[pos]) * scale[pos],
                                                          _row(f, dim, at, count, rows[neg]) * scale[neg]))

    put(3, n - 6, 0, 1)
    if flags >> (2 * axis) & 1:
        for r, (p, q) in enumerate(((2, 2), (2, 3), (0, 4))):
            put(3 + r, 1, p, q)
    if flags >> (2 * axis + 1) & 1:
        for r, (p, q) in enumerate(((2, 1), (3, 4), (4, 4))):
            put(n - 6 + r, 1, p, q)
    return out


_SYM = {(0, 0): 0, (0, 1): 1, (0, 2): 2, (1, 1): 3, (1, 2): 4, (2, 2): 5}
R3 = range(3)


def _s(i, j):
    return _SYM[(min(i, j), max(i, j))]


def _total(terms):
    acc = None
    for t in terms:
        acc = t if acc is None else acc + t
    return acc


class _Geometry:
    """What the right-hand side and the constraints share, at the interior points of same-shaped blocks."""

    def __init__(self, f, h, flags, second):
        inner = (slice(None), slice(3, -3), slice(3, -3), slice(3, -3))
        self.inner = inner
        self.u = [g[inner] for g in f]
        grad = [[_d1(g, a, h[a], flags) for a in R3] for g in f]
        self.d = [[g[a][inner].contiguous() for a in R3] for g in grad]
        self.dd = {}
        for v in second:
            m = {(0, 1): _d1(grad[v][0], 1, h[1], flags), (0, 2): _d1(grad[v][0], 2, h[2], flags),
                 (1, 2): _d1(grad[v][1], 2, h[2], flags)}
            for a in R3:
                m[(a, a)] = _d2(f[v], a, h[a], flags)
            self.dd[v] = {k: t[inner].contiguous() for k, t in m.items()}
        del grad
        u, d = self.u, self.d
        self.chi, self.K, self.alpha = u[1], u[2], u[0]
        self.dchi = d[1]
        gt = self.gt = [[u[12 + _s(i, j)] for j in R3] for i in R3]
        self.At = [[u[18 + _s(i, j)] for j in R3] for i in R3]
        det = gt[0][0] * (gt[1][1] * gt[2][2] - gt[1][2] ** 2) - gt[0][1] * (gt[0][1] * gt[2][2] - gt[1][2] * gt[0][2]) \
            + gt[0][2] * (gt[0][1] * gt[1][2] - gt[1][1] * gt[0][2])
        up = {}
        for i, j in _SYM:
            a, b = [x for x in R3 if x != i], [x for x in R3 if x != j]
            up[(i, j)] = (gt[a[0]][b[0]] * gt[a[1]][b[1]] - gt[a[0]][b[1]] * gt[a[1]][b[0]]) * ((-1) ** (i + j)) / det
        g = self.igt = [[up[(min(i, j), max(i, j))] for j in R3] for i in R3]
        dg = lambda a, i, j: d[12 + _s(i, j)][a]  # noqa: E731
        C1 = self.C1 = [[[0.5 * (dg(j, k, i) + dg(i, k, j) - dg(k, i, j)) for j in R3] for i in R3] for k in R3]
        C2 = self.C2 = [[[None] * 3 for _ in R3] for _ in R3]
        for k in R3:
            for i, j in _SYM:
                C2[k][i][j] = C2[k][j][i] = _total(g[k][m] * C1[m][i][j] for m in R3)
        self.Cal = [_total(g[i][j] * C2[k][i][j] for i in R3 for j in R3) for k in R3]
        self.R = self._ricci()

    def _ricci(self):
        d, g, gt, C1, C2, chi, dchi = self.d, self.igt, self.gt, self.C1, self.C2, self.chi, self.dchi
        dGt = lambda i, k: d[3 + k][i]  # noqa: E731
        d2chi = lambda i, j: self.dd[1][(min(i, j), max(i, j))]  # noqa: E731
        lap = _total(g[k][m] * (d2chi(k, m) - 1.5 / chi * dchi[k] * dchi[m]) for k in R3 for m in R3) \
            - _total(self.Cal[m] * dchi[m] for m in R3)
        R = {}
        for i, j in _SYM:
            dd = self.dd[12 + _s(i, j)]
            t = _total(-0.5 * g[k][m] * dd[(min(k, m), max(k, m))] for k in R3 for m in R3)
            t = t + 0.5 * _total(gt[k][i] * dGt(j, k) + gt[k][j] * dGt(i, k) + self.Cal[k] * (C1[i][j][k] + C1[j][i][k])
                                 for k in R3)
            for l in R3:
                for m in R3:
                    t = t + g[l][m] * _total(C2[k][l][i] * C1[j][k][m] + C2[k][l][j] * C1[i][k][m] + C2[k][i][m] * C1[k][l][j]
                                             for k in R3)
            x = d2chi(i, j) - _total(C2[k][i][j] * dchi[k] for k in R3) - 0.5 / chi * dchi[i] * dchi[j] + gt[i][j] * lap
            R[(i, j)] = t + 0.5 / chi * x
        return [[R[(min(i, j), max(i, j))] for j in R3] for i in R3]

    def a_up(self):
        """A with both indices up."""
        g, A = self.igt, self.At
        half = [[_total(g[i][k] * A[k][j] for k in R3) for j in R3] for i in R3]  # A^i_j
        return half, [[_total(half[i][k] * g[k][j] for k in R3) for j in R3] for i in R3]


def _rhs_group(f, h, flags, x, prm, upwind):
    """24 right-hand sides (without dissipation) at the interior points; `f`: [24] of [nb, nz, ny, nx]."""
    G = _Geometry(f, h, flags, (12, 13, 14, 15, 16, 17, 1, 0, 6, 7, 8))
    u, d, g, gt, A, C2, alpha, chi, K = G.u, G.d, G.igt, G.gt, G.At, G.C2, G.alpha, G.chi, G.K
    beta = u[6:9]
    if upwind:
        adv = [_total(beta[a] * _upwind(f[v], a, h[a], flags, f[6 + a])[G.inner] for a in R3) for v in range(NUM_VARS)]
    else:
        adv = [_total(beta[a] * d[v][a] for a in R3) for v in range(NUM_VARS)]
    r = torch.sqrt(x[0] * x[0] + x[1] * x[1] + x[2] * x[2])
    eta = torch.where(r >= prm.eta_r0, prm.eta_const * (prm.eta_r0 / r) ** prm.eta_damping_exp, torch.full_like(r, prm.eta_const))
    lam, lf = [float(v) for v in prm.lambda_], [float(v) for v in prm.lambda_f]
    out = [None] * NUM_VARS
    div = _total(d[6 + a][a] for a in R3)
    db = lambda a, i: d[6 + i][a]  # noqa: E731
    half, Aup = G.a_up()
    AA = _total(A[i][j] * Aup[i][j] for i in R3 for j in R3)
    da = d[0]
    low = _total(g[0][m] * G.dchi[m] for m in R3), _total(g[1][m] * G.dchi[m] for m in R3), _total(g[2][m] * G.dchi[m] for m in R3)
    out[0] = lam[0] * adv[0] - 2 * alpha * K
    out[1] = adv[1] + (2.0 / 3.0) * chi * (alpha * K - div)
    DD = {}
    for i, j in _SYM:
        c3 = [C2[k][i][j] - 0.5 / chi * ((G.dchi[i] if k == j else 0.0) + (G.dchi[j] if k == i else 0.0) - gt[i][j] * low[k])
              for k in R3]
        DD[(i, j)] = G.dd[0][(i, j)] - _total(c3[k] * da[k] for k in R3)
    DDs = lambda i, j: DD[(min(i, j), max(i, j))]  # noqa: E731
    out[2] = adv[2] - chi * _total(g[i][j] * DDs(i, j) for i in R3 for j in R3) + alpha * (K * K / 3.0 + AA)
    X = {(i, j): alpha * G.R[i][j] - DDs(i, j) for i, j in _SYM}
    trace = _total(g[i][j] * X[(min(i, j), max(i, j))] for i in R3 for j in R3)
    for i, j in _SYM:
        lie = lambda T: _total(T[k][j] * db(i, k) + T[i][k] * db(j, k) for k in R3) - (2.0 / 3.0) * T[i][j] * div  # noqa: E731
        out[12 + _s(i, j)] = adv[12 + _s(i, j)] + lie(gt) - 2 * alpha * A[i][j]
        AikAkj = _total(A[i][k] * half[k][j] for k in R3)
        out[18 + _s(i, j)] = adv[18 + _s(i, j)] + lie(A) + chi * (X[(i, j)] - gt[i][j] * trace / 3.0) \
            + alpha * (K * A[i][j] - 2 * AikAkj)
    for i in R3:
        bb = lambda j, k, m: G.dd[6 + m][(min(j, k), max(j, k))]  # noqa: E731
        t = adv[3 + i] - _total(G.Cal[j] * db(j, i) for j in R3) + (2.0 / 3.0) * G.Cal[i] * div
        t = t + _total(g[j][k] * bb(j, k, i) for j in R3 for k in R3) + _total(g[i][j] * bb(j, k, k) for j in R3 for k in R3) / 3.0
        t = t - 2 * _total(Aup[i][j] * da[j] for j in R3)
        t = t + 2 * alpha * (_total(C2[i][j][k] * Aup[j][k] for j in R3 for k in R3)
                             - 1.5 / chi * _total(Aup[i][j] * G.dchi[j] for j in R3)
                             - (2.0 / 3.0) * _total(g[i][j] * d[2][j] for j in R3))
        out[3 + i] = t
        out[6 + i] = 0.75 * (lf[0] + lf[1] * alpha) * u[9 + i] + lam[1] * adv[6 + i]
        out[9 + i] = t - eta * u[9 + i] + lam[2] * adv[9 + i] - lam[3] * adv[3 + i]
    if flags:  # Sommerfeld values on the flagged face planes
        face = torch.zeros_like(r, dtype=torch.bool)
        for a in R3:
            if flags >> (2 * a) & 1:
                face.narrow(3 - a, 0, 1).fill_(True)
            if flags >> (2 * a + 1) & 1:
                face.narrow(3 - a, face.shape[3 - a] - 1, 1).fill_(True)
        for v in range(NUM_VARS):
            fall = 2.0 if 3 <= v <= 5 or v >= 18 else 1.0
            limit = 1.0 if v in (0, 1, 12, 15, 17) else 0.0
            val = -(x[0] * d[v][0] + x[1] * d[v][1] + x[2] * d[v][2] + fall * (u[v] - limit)) / r
            out[v] = torch.where(face, val, out[v])
    return out


def _constraints_group(f, h, flags):
    G = _Geometry(f, h, flags, (12, 13, 14, 15, 16, 17, 1))
    g, A, d = G.igt, G.At, G.d
    half, Aup = G.a_up()
    out = [G.chi * _total(g[i][j] * G.R[i][j] for i in R3 for j in R3)
           - _total(A[i][j] * Aup[i][j] for i in R3 for j in R3) + (2.0 / 3.0) * G.K * G.K]
    for i in R3:
        t = -(2.0 / 3.0) * d[2][i] - _total(G.u[3 + k] * A[k][i] for k in R3)
        for j in R3:
            for k in R3:
                t = t + g[j][k] * (d[18 + _s(k, i)][j] - _total(G.C2[m][i][j] * A[k][m] for m in R3)
                                   - 1.5 / G.chi * A[i][j] * G.dchi[k])
        out.append(t)
    return out


def _evaluate(u, blocks, put, prm=None, upwind=False):
    """Calls put(blocks of one shape, their element numbers [nb, points], values) for every block: the
    24 right-hand sides with `prm`, else the four constraints."""
    groups = {}
    for b in blocks:
        groups.setdefault((tuple(b.sz), b.bflag), []).append(b)
    dev = u.device
    for ((nx, ny, nz), flags), group in groups.items():
        step = max(1, 2_400_000 // (nx * ny * nz))
        shape = (nz, ny, nx)
        for s in range(0, len(group), step):
            part = group[s:s + step]
            at = torch.tensor([b.offset for b in part], device=dev)[:, None] + torch.arange(nx * ny * nz, device=dev)
            f = [u[v][at.reshape(-1)].reshape(len(part), *shape) for v in range(NUM_VARS)]
            col = lambda vals: torch.tensor(vals, dtype=torch.float64, device=dev).reshape(-1, 1, 1, 1)  # noqa: E731
            h = [col([b.h[a] for b in part]) for a in R3]
            inner = at.reshape(len(part), *shape)[:, 3:-3, 3:-3, 3:-3]
            if prm is None:
                put(part, inner, _constraints_group(f, h, flags))
                continue
            x = []
            for a, n in enumerate((nx, ny, nz)):
                line = torch.arange(3, n - 3, dtype=torch.float64, device=dev)
                view = [1, 1, 1, 1]
                view[3 - a] = n - 6
                x.append((col([b.pmin[a] for b in part]) + line.reshape(view) * h[a]).expand(inner.shape))
            vals = _rhs_group(f, h, flags, x, prm, upwind)
            for v in range(NUM_VARS):
                ko = _ko(f[v], 0, h[0], flags) + _ko(f[v], 1, h[1], flags) + _ko(f[v], 2, h[2], flags)
                vals[v] = vals[v] + prm.ko_sigma * ko[:, 3:-3, 3:-3, 3:-3]
            put(part, inner, vals)


def _rhs(u, blocks, prm, upwind):
    rhs = torch.zeros_like(u)

    def put(part, at, vals):
        for v in range(NUM_VARS):
            rhs[v].index_copy_(0, at.reshape(-1), vals[v].reshape(-1))

    _evaluate(u, blocks, put, prm, upwind)
    return rhs


def exact(case, seed, device="cuda"):
    blocks, total = _layout(case, seed)
    u = _fields(blocks, total, seed, device)
    prm = _params(case)
    if case["kind"] == "constraints":
        con = torch.zeros((4, total), dtype=torch.float64, device=device)
        norms = torch.zeros((len(blocks), 8), dtype=torch.float64, device=device)
        number = {b.offset: i for i, b in enumerate(blocks)}

        def put(part, at, vals):
            rows = torch.tensor([number[b.offset] for b in part], device=device)
            for c in range(4):
                con[c].index_copy_(0, at.reshape(-1), vals[c].reshape(-1))
                flat = vals[c].reshape(len(part), -1)
                norms[rows, c] = (flat * flat).sum(1)
                norms[rows, 4 + c] = flat.abs().max(1).values

        _evaluate(u, blocks, put)
        return {"con": con, "norms": norms}
    if case["kind"] != "rk4":
        rhs = _rhs(u, blocks, prm, case.get("upwind", False))
        return rhs.cpu().numpy() if case["kind"] == "dropin" else rhs
    dt = _dt(blocks)
    k1 = _rhs(u, blocks, prm, False)
    acc = k1 * (dt / 6)
    k = _rhs(u + k1 * (dt / 2), blocks, prm, False)
    acc += k * (dt / 3)
    k = _rhs(u + k * (dt / 2), blocks, prm, False)
    acc += k * (dt / 3)
    k = _rhs(u + k * dt, blocks, prm, False)
    return u + acc + k * (dt / 6)
