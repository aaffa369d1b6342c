"""The solver's work as its users have it done, as timed cases.

A case is one of three programs:

``step``   new values on a known pattern (already on the GPU, in the matrix's own CSC
           order) -> bcsc -> numerical factorization -> solve of nrhs right-hand sides
           -> with an FP32 factor the FP64 refinement to 1e-12: the loop of a simulation
           that refactors every time step, and of the benchmark.
``solve``  right-hand sides against a factor that stays resident (the serving program);
           with an FP32 factor again with its refinement.
``host``   ``step`` with host values and host vectors, the calls of PaStiX's own task
           API (numfact, solve, refine on numpy arrays).

The matrices are the grid problems of the benchmark and the tests (7- and 27-point
Laplacians, the convection-diffusion LU, shifted indefinite Laplacians in 3D and in 2D
batches), with the diagonal scaling d_i uniform in [0.9, 1.1] of the serving workload, so
that every seed has other values.  The analysis below (geometric nested dissection,
symbolic factorization, cblks split at 320 columns) stands for the saved analysis that
such a program starts from; it depends on the grid alone.  Right-hand sides are
b = A x_true with x_true uniform in [-1, 1], so the exact result is x_true.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from pastix_b200 import native
from pastix_b200.batch import concat_structures
from pastix_b200.refhost import BCSC, SolverStructure

MAX_WIDTH = 320   # IPARM_MAX_BLOCKSIZE
LEAF_CELLS = 9
FACTO_ID = {"potrf": 0, "sytrf": 1, "getrf": 2}


# ---------------------------------------------------------------- the cases

def listed():
    return [
        # the smallest call of the tests and the smoke run: launches and host latency
        dict(name="step_potrf7_10x9x11_fp64", kind="step", facto="potrf", points=7, nx=10, ny=9, nz=11, prec="fp64",
             nrhs=1, shift=0.0),
        # the first workload: plain FP64 Cholesky of the 20^3 7-point Laplacian, one right-hand side
        dict(name="step_potrf7_20_fp64", kind="step", facto="potrf", points=7, nx=20, ny=20, nz=20, prec="fp64",
             nrhs=1, shift=0.0),
        # the headline workload, drop-in FP64 path
        dict(name="step_potrf27_80_fp64", kind="step", facto="potrf", points=27, nx=80, ny=80, nz=80, prec="fp64",
             nrhs=16, shift=1e-3),
        # the headline workload, fastest mixed path with CG
        dict(name="step_potrf27_80_bf16x3", kind="step", facto="potrf", points=27, nx=80, ny=80, nz=80,
             prec="bf16x3", nrhs=16, shift=1e-3),
        # the other tensor-core path at a ragged size and an odd number of right-hand sides
        dict(name="step_potrf27_61x45x52_tf32x3", kind="step", facto="potrf", points=27, nx=61, ny=45, nz=52,
             prec="tf32x3", nrhs=5, shift=1e-3),
        # the LU workload: 64^3 convection-diffusion, static pivoting, GMRES
        dict(name="step_getrf7_64_tf32x3", kind="step", facto="getrf", points=7, nx=64, ny=64, nz=64, prec="tf32x3",
             nrhs=8, shift=0.0),
        # LU in FP64, ragged, through host arrays
        dict(name="host_getrf7_37x30x41_fp64", kind="host", facto="getrf", points=7, nx=37, ny=30, nz=41,
             prec="fp64", nrhs=3, shift=0.0),
        # indefinite 3D LDL^T with an FP32 factor
        dict(name="step_sytrf7_44x40x39_tf32x3", kind="step", facto="sytrf", points=7, nx=44, ny=40, nz=39,
             prec="tf32x3", nrhs=4, shift=-0.05),
        # the batched workload: a forest of 2D LDL^T systems, sides log-uniform in [16, 128]
        dict(name="batch_sytrf5_512_fp32", kind="step", facto="sytrf", points=5, nx=16, ny=128, nz=512, prec="fp32",
             nrhs=1, shift=-0.02),
        # serving: resident FP32 factor, one batch of requests
        dict(name="solve_potrf7_100_tf32x3_r64", kind="solve", facto="potrf", points=7, nx=100, ny=100, nz=100,
             prec="tf32x3", nrhs=64, shift=0.0),
        # serving on the FP64 factor: a full batch of slots, and a single small request
        dict(name="solve_potrf7_100_fp64_r256", kind="solve", facto="potrf", points=7, nx=100, ny=100, nz=100,
             prec="fp64", nrhs=256, shift=0.0),
        dict(name="solve_potrf7_33x41x37_fp64_r1", kind="solve", facto="potrf", points=7, nx=33, ny=41, nz=37,
             prec="fp64", nrhs=1, shift=0.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    form = rng.choice(["potrf27", "potrf7", "getrf", "sytrf", "batch", "solve", "solve"])
    if form == "batch":
        lo = rng.randint(16, 40)
        return dict(kind="step", facto="sytrf", points=5, nx=lo, ny=rng.randint(lo, 128), nz=_log_int(rng, 16, 512),
                    prec=rng.choice(["fp32", "fp64"]), nrhs=rng.choice([1, 1, 3]), shift=-0.02)
    top = {"potrf27": 80, "potrf7": 96, "getrf": 64, "sytrf": 48, "solve": 96}[form]
    side = math.exp(rng.uniform(math.log(9), math.log(top)))
    nx, ny, nz = (max(6, min(top, int(round(side * math.exp(rng.uniform(-0.25, 0.25)))))) for _ in range(3))
    points = 27 if form == "potrf27" or (form == "solve" and max(nx, ny, nz) <= 64 and rng.random() < 0.5) else 7
    facto = {"potrf27": "potrf", "potrf7": "potrf", "getrf": "getrf", "sytrf": "sytrf"}.get(form)
    if facto is None:
        facto = "potrf" if max(nx, ny, nz) > 48 else rng.choice(["potrf", "potrf", "getrf", "sytrf"])
        points = 7 if facto == "getrf" else points
    kind = "solve" if form == "solve" else rng.choice(["step", "step", "step", "host"])
    nrhs = _log_int(rng, 1, 256) if kind == "solve" else _log_int(rng, 1, 32)
    shift = -0.05 if facto == "sytrf" else 1e-3 if points == 27 else 0.0
    return dict(kind=kind, facto=facto, points=points, nx=nx, ny=ny, nz=nz,
                prec=rng.choice(["fp64", "fp64", "tf32x3", "bf16x3", "fp32"]), nrhs=nrhs, shift=shift)


# ---------------------------------------------------------------- analysis

def _boxes(nx, ny, nz):
    """Nested dissection of the grid: per node (post-order) its box and the cells it
    eliminates (a separator plane, or the whole box of a leaf)."""
    boxes, parts = [], []

    def rec(b):
        d = [b[1] - b[0], b[3] - b[2], b[5] - b[4]]
        a = d.index(max(d))
        if d[0] * d[1] * d[2] <= LEAF_CELLS or d[a] < 3:
            boxes.append(b)
            parts.append(b)
            return
        m = (b[2 * a] + b[2 * a + 1]) // 2
        lo, hi, mid = list(b), list(b), list(b)
        lo[2 * a + 1] = m
        hi[2 * a] = m + 1
        mid[2 * a], mid[2 * a + 1] = m, m + 1
        rec(tuple(lo))
        rec(tuple(hi))
        boxes.append(b)
        parts.append(tuple(mid))

    rec((0, nx, 0, ny, 0, nz))
    return np.array(boxes, dtype=np.int64), np.array(parts, dtype=np.int64)


@functools.lru_cache(maxsize=None)
def _inner_order(dx, dy, dz):
    """Order of a separator's (or leaf's) cells: halves first, then the cut between
    them, so that the boxes beside it touch few row intervals."""
    out = []

    def rec(b):
        d = [b[1] - b[0], b[3] - b[2], b[5] - b[4]]
        a = d.index(max(d))
        if d[a] < 3:
            out.extend((z * dy + y) * dx + x for z in range(b[4], b[5]) for y in range(b[2], b[3])
                       for x in range(b[0], b[1]))
            return
        m = (b[2 * a] + b[2 * a + 1]) // 2
        for lo, hi in ((b[2 * a], m), (m + 1, b[2 * a + 1]), (m, m + 1)):
            c = list(b)
            c[2 * a], c[2 * a + 1] = lo, hi
            rec(tuple(c))

    rec((0, dx, 0, dy, 0, dz))
    return np.array(out, dtype=np.int64)


def _cells(boxes, nx, ny):
    """(box index, cell) of every cell of every box, box after box."""
    dx, dy, dz = boxes[:, 1] - boxes[:, 0], boxes[:, 3] - boxes[:, 2], boxes[:, 5] - boxes[:, 4]
    size = dx * dy * dz
    start = np.cumsum(size) - size
    own = np.repeat(np.arange(len(boxes)), size)
    loc = np.arange(own.size) - start[own]
    q = loc // dx[own]
    x = boxes[own, 0] + loc - q * dx[own]
    z = q // dy[own]
    y = boxes[own, 2] + q - z * dy[own]
    return own, x + nx * (y + ny * (boxes[own, 4] + z))


@functools.lru_cache(maxsize=4)
def _structure(nx, ny, nz, points, facto):
    """Ordering and SolverMatrix tables of the grid."""
    n = nx * ny * nz
    boxes, parts = _boxes(nx, ny, nz)
    nn = len(boxes)
    dims = parts[:, 1::2] - parts[:, 0::2]
    width = dims.prod(axis=1)
    first = np.cumsum(width) - width
    _, cell = _cells(parts, nx, ny)
    peri = np.empty(n, dtype=np.int64)
    shapes, which = np.unique(dims, axis=0, return_inverse=True)
    for i, (dx, dy, dz) in enumerate(shapes):
        o = _inner_order(int(dx), int(dy), int(dz))
        at = first[which.ravel() == i][:, None]
        peri[at + np.arange(o.size)] = cell[at + o]
    perm = np.empty(n, dtype=np.int64)
    perm[peri] = np.arange(n)

    # rows below each node: the grid cells beside its box
    lim = np.array([nx, ny, nz])
    slabs = []
    grown = boxes.copy()
    if points == 27:
        grown[:, 0::2] = np.maximum(boxes[:, 0::2] - 1, 0)
        grown[:, 1::2] = np.minimum(boxes[:, 1::2] + 1, lim)
    for a in range(3):
        for side in (0, 1):
            s = boxes.copy()
            s[:, :2 * a] = grown[:, :2 * a]
            s[:, 2 * a] = boxes[:, 2 * a] - 1 if side == 0 else boxes[:, 2 * a + 1]
            s[:, 2 * a + 1] = s[:, 2 * a] + 1
            ok = (s[:, 2 * a] >= 0) & (s[:, 2 * a] < lim[a])
            slabs.append((np.nonzero(ok)[0], s[ok]))
    node = np.concatenate([s[0] for s in slabs])
    own, cell = _cells(np.concatenate([s[1] for s in slabs]), nx, ny)
    key = np.sort(node[own] * n + perm[cell])
    own, row = key // n, key % n

    # cblks: nodes wider than MAX_WIDTH in equal parts
    npart = -(-width // MAX_WIDTH)
    c0 = np.cumsum(npart) - npart
    cn = int(npart.sum())
    cnode = np.repeat(np.arange(nn), npart)
    cpart = np.arange(cn) - c0[cnode]
    fcol = first[cnode] + cpart * width[cnode] // npart[cnode]
    lcol = np.concatenate([fcol[1:], [n]]) - 1
    col2cblk = np.repeat(np.arange(cn), lcol - fcol + 1)

    # row intervals of every node, cut where the facing cblk changes
    f = col2cblk[row]
    new = np.ones(row.size, dtype=bool)
    new[1:] = (own[1:] != own[:-1]) | (row[1:] != row[:-1] + 1) | (f[1:] != f[:-1])
    at = np.nonzero(new)[0]
    i_lo, i_hi, i_f = row[at], row[np.concatenate([at[1:], [row.size]]) - 1] if at.size else row[at], f[at]
    icnt = np.bincount(own[at], minlength=nn)
    i0 = np.cumsum(icnt) - icnt

    later = npart[cnode] - 1 - cpart
    nblk = 1 + later + icnt[cnode]
    fblok = np.concatenate([[0], np.cumsum(nblk)])
    bn = int(fblok[-1])
    bown = np.repeat(np.arange(cn), nblk)
    loc = np.arange(bn) - fblok[bown]
    inside = loc <= later[bown]
    bf = np.where(inside, bown + loc, 0)
    frow, lrow = fcol[bf].copy(), lcol[bf].copy()
    out = ~inside
    ii = i0[cnode[bown[out]]] + loc[out] - 1 - later[bown[out]]
    frow[out], lrow[out], bf[out] = i_lo[ii], i_hi[ii], i_f[ii]
    rows = lrow - frow + 1
    roff = np.cumsum(rows) - rows
    roff -= roff[fblok[bown]]
    stride = np.add.reduceat(rows, fblok[:-1])
    ncol = lcol - fcol + 1

    off = loc > 0
    brow = np.nonzero(off)[0]
    brow = brow[np.argsort(bf[brow], kind="stable")]
    browcnt = np.bincount(bf[off], minlength=cn)
    brownum = np.concatenate([[0], np.cumsum(browcnt)])
    browind = np.full(bn + 1, -1)
    browind[brow] = np.arange(brow.size)
    m = (stride - ncol).astype(float)
    w = ncol.astype(float)
    flops = float((w * m * m + m * w * (w + 1) + w * (w + 1) * (2 * w + 1) / 6).sum())
    if facto == "getrf":
        flops *= 2
    app = lambda a, v: np.ascontiguousarray(np.concatenate([a, [v]]), dtype=np.int64)  # noqa: E731
    return SolverStructure(
        n, cn, bn, int(brow.size), int((stride * ncol).sum()), FACTO_ID[facto], app(fcol, n), app(lcol, n),
        fblok.astype(np.int64), app(stride, 0), app(fcol, n), brownum.astype(np.int64), brownum.astype(np.int64),
        np.zeros(cn + 1, np.int32), app(frow, n), app(lrow, n), app(bown, cn + 1), app(bf, cn + 1),
        app(roff * ncol[bown], 0), browind.astype(np.int64), brow.astype(np.int64), perm, peri, flops, cn)


def _offsets(points):
    r = (-1, 0, 1)
    if points == 27:
        return [(i, j, k) for k in r for j in r for i in r]
    if points == 5:
        return [(0, -1, 0), (-1, 0, 0), (0, 0, 0), (1, 0, 0), (0, 1, 0)]
    return [(0, 0, -1), (0, -1, 0), (-1, 0, 0), (0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1)]


@functools.lru_cache(maxsize=4)
def _pattern(nx, ny, nz, points, facto, device="cpu"):
    """The matrix's own CSC (the lower triangle when symmetric): row and column of
    every value; and its bcsc: column pointers, rows, and the value each entry holds."""
    st = _structure(nx, ny, nz, points, facto)
    n = st.n
    c = torch.arange(n, device=device)
    x, y, z = c % nx, c // nx % ny, c // (nx * ny)
    offs = _offsets(points)
    lin = torch.tensor([i + nx * (j + ny * k) for i, j, k in offs], device=device)
    ok = torch.stack([(x + i >= 0) & (x + i < nx) & (y + j >= 0) & (y + j < ny) & (z + k >= 0) & (z + k < nz)
                      for i, j, k in offs], dim=1)
    nb = torch.where(ok, c[:, None] + lin, 0)
    k = len(offs)
    mine = ok.clone()
    if facto != "getrf":
        mine[:, :k // 2] = False
    idx = (torch.cumsum(mine.reshape(-1), 0) - 1).reshape(n, k)
    flip = torch.arange(k - 1, -1, -1, device=device)
    back = idx[nb, flip[None, :].expand(n, k)]  # the entry of the transposed position
    low = idx if facto == "getrf" else torch.where(mine, idx, back)
    peri = torch.from_numpy(st.peritab).to(device)
    perm = torch.from_numpy(st.permtab).to(device)
    okp = ok[peri]
    rows, order = torch.sort(torch.where(okp, perm[nb[peri]], n), dim=1)
    keep = rows < n
    take = lambda t: torch.gather(t[peri], 1, order)[keep].cpu().numpy()  # noqa: E731
    colptr = torch.cat([torch.zeros(1, dtype=torch.int64, device=device), torch.cumsum(keep.sum(1), 0)])
    return dict(n=n, nnz=int(mine.sum()), row=nb[mine], col=c[:, None].expand(n, k)[mine],
                slot=torch.arange(k, device=device).expand(n, k)[mine], colptr=colptr.cpu().numpy(),
                rowtab=rows[keep].cpu().numpy(), lmap=take(low), umap=take(back) if facto == "getrf" else None)


# ---------------------------------------------------------------- values

def _stencil(case):
    """Off-diagonal -1 everywhere; the diagonal is the number of neighbours plus the
    shift (2D and 3D alike, an indefinite shift for LDL^T)."""
    return float(case["points"] - 1) + case["shift"]


def _system(case, dims, rng, device):
    """Values in CSC order, x_true and b of one grid (deterministic from rng)."""
    nx, ny, nz = dims
    p = _pattern(nx, ny, nz, case["points"], case["facto"], device)
    n = p["n"]
    dev = lambda a: torch.from_numpy(a).to(device)  # noqa: E731
    xt = dev(rng.uniform(-1.0, 1.0, (case["nrhs"], n)))
    offs = _offsets(case["points"])
    g = (case["nrhs"], nz, ny, nx)

    def shifted(v, off):  # v of the neighbour at off, 0 outside the grid
        out = torch.zeros_like(v)
        src, dst = [slice(None)], [slice(None)]
        for o, m in zip(off[::-1], (nz, ny, nx)):
            dst.append(slice(max(0, -o), m - max(0, o)))
            src.append(slice(max(0, o), m - max(0, -o)))
        out[tuple(dst)] = v[tuple(src)]
        return out

    if case["facto"] == "getrf":
        # upwind convection-diffusion: row i has -1 towards larger neighbours,
        # -1 - h v_d(i) towards smaller ones, 6 + h sum v on the diagonal
        h = 1.0 / (max(dims) + 1)
        hv = dev(rng.uniform(0.0, 50.0, (3, n)) * h)
        diag = 6.0 + hv.sum(0)
        axis = [next((a for a in range(3) if o[a]), 0) for o in offs]
        ax = torch.tensor(axis, device=device)[p["slot"]]
        below = p["row"] > p["col"]  # the row's smaller neighbour
        vals = torch.where(p["row"] == p["col"], diag[p["row"]], torch.where(below, -1.0 - hv[ax, p["row"]], -1.0))
        v = xt.reshape(g)
        b = diag.reshape(1, nz, ny, nx) * v
        for a, o in zip(axis, offs):
            if sum(o) > 0:
                b -= shifted(v, o)
            elif sum(o) < 0:
                b -= (1.0 + hv[a]).reshape(1, nz, ny, nx) * shifted(v, o)
        return vals, xt, b.reshape(case["nrhs"], n)
    d = dev(rng.uniform(0.9, 1.1, n))
    vals = torch.where(p["row"] == p["col"], _stencil(case) * d[p["row"]], -d[p["row"]]) * d[p["col"]]
    v = (xt * d).reshape(g)
    b = _stencil(case) * v
    for o in offs:
        if any(o):
            b -= shifted(v, o)
    return vals, xt, b.reshape(case["nrhs"], n) * d


@functools.lru_cache(maxsize=4)
def _batch_sides(lo, hi, nsys):
    """Sides of a batch's systems, log-uniform in [lo, hi] (a fixed program's systems)."""
    u = (np.arange(nsys) + 0.5) / nsys
    return np.random.default_rng(7).permutation(np.floor(lo * ((hi + 1) / lo) ** u).astype(int).clip(lo, hi))


@functools.lru_cache(maxsize=2)
def _batch_structure(lo, hi, nsys):
    sides = _batch_sides(lo, hi, nsys)
    sts = [_structure_of_side(int(s)) for s in sides]
    st, sys_cblk = concat_structures(sts)
    ps = [_pattern_of_side(int(s)) for s in sides]
    n0 = np.concatenate([[0], np.cumsum([p["n"] for p in ps])])
    v0 = np.concatenate([[0], np.cumsum([p["nnz"] for p in ps])])
    e0 = np.concatenate([[0], np.cumsum([p["colptr"][-1] for p in ps])])
    return dict(st=st, sys_cblk=sys_cblk, nnz=int(v0[-1]),
                colptr=np.concatenate([p["colptr"][:-1] + e for p, e in zip(ps, e0)] + [[e0[-1]]]),
                rowtab=np.concatenate([p["rowtab"] + o for p, o in zip(ps, n0)]),
                lmap=np.concatenate([p["lmap"] + o for p, o in zip(ps, v0)]))


@functools.lru_cache(maxsize=128)
def _structure_of_side(s):
    return _structure(s, s, 1, 5, "sytrf")


@functools.lru_cache(maxsize=128)
def _pattern_of_side(s):
    return _pattern(s, s, 1, 5, "sytrf")


def _batch_values(case, rng):
    """The batch's values and vectors, system after system (on the host: small grids)."""
    sides = _batch_sides(case["nx"], case["ny"], case["nz"])
    vals, xts, bs = [], [], []
    for s in sides:
        s = int(s)
        p = _pattern_of_side(s)
        d = rng.uniform(0.9, 1.1, (s, s))
        sigma = rng.uniform(0.0, 1.0) * case["shift"] * 8.0  # of the largest eigenvalue
        df = d.ravel()
        r, c = p["row"].numpy(), p["col"].numpy()
        vals.append(np.where(r == c, 4.0 + sigma, -1.0) * df[r] * df[c])
        xt = rng.uniform(-1.0, 1.0, (case["nrhs"], s, s))
        v = np.zeros((case["nrhs"], s + 2, s + 2))
        v[:, 1:-1, 1:-1] = xt * d
        b = (4.0 + sigma) * v[:, 1:-1, 1:-1]
        b = b - v[:, :-2, 1:-1] - v[:, 2:, 1:-1] - v[:, 1:-1, :-2] - v[:, 1:-1, 2:]
        xts.append(xt.reshape(case["nrhs"], -1))
        bs.append((b * d).reshape(case["nrhs"], -1))
    return tuple(torch.from_numpy(np.concatenate(a, axis=-1)) for a in (vals, xts, bs))


def _is_batch(case):
    return case["points"] == 5


def _inputs(case, seed, device):
    rng = np.random.default_rng(seed)
    if _is_batch(case):
        return tuple(t.to(device) for t in _batch_values(case, rng))
    return _system(case, (case["nx"], case["ny"], case["nz"]), rng, device)


# ---------------------------------------------------------------- the program

def _analysis(case, device="cuda"):
    if _is_batch(case):
        return _batch_structure(case["nx"], case["ny"], case["nz"])
    key = (case["nx"], case["ny"], case["nz"], case["points"], case["facto"])
    return dict(_pattern(*key, device), st=_structure(*key))


def _eps_magn(case):
    """DPARM_EPSILON_MAGN_CTRL: static pivoting at 1e-8 ||A|| for LU; LDL^T systems in
    FP32 use 1e-6 ||A||, the default (0) elsewhere."""
    return {"getrf": 1e-8, "sytrf": 1e-6 if case["prec"] != "fp64" else 0.0}.get(case["facto"], 0.0)


def prepare(case, seed):
    a = _analysis(case)
    st = a["st"]
    stream = torch.cuda.Stream()
    vals, _, b = _inputs(case, seed, "cuda")
    torch.cuda.synchronize()
    s = native.Solver(st, case["facto"], case["prec"], stream=stream.cuda_stream)
    if _is_batch(case):
        s.batch_set(a["sys_cblk"])
    zeros = np.zeros(a["rowtab"].size)
    s.bcsc_load(BCSC(st.n, a["colptr"], a["rowtab"], zeros, zeros if case["facto"] == "getrf" else None, 0.0))
    s.spm_map(a["nnz"], a["lmap"], a.get("umap"))
    state = dict(case=case, s=s, stream=stream, n=st.n)
    if case["kind"] == "host":
        state["values"] = vals.cpu().numpy()
        state["b"] = np.asfortranarray(b.cpu().numpy().T)
        return state
    state["values"], state["b"] = vals, b
    state["x"] = torch.empty_like(b)
    if case["kind"] == "solve":
        s.spm_values_device(vals.data_ptr())
        s.numfact(_eps_magn(case))
    torch.cuda.synchronize()
    return state


def run(state):
    case, s = state["case"], state["s"]
    method = "cg" if case["facto"] == "potrf" else "gmres"
    if case["kind"] == "host":
        s.spm_values(state["values"])
        s.numfact(_eps_magn(case))
        x = s.solve(state["b"])
        if case["prec"] != "fp64":
            x, _, _ = s.refine(state["b"], x, method)
        return x
    with torch.cuda.stream(state["stream"]):
        if case["kind"] == "step":
            s.spm_values_device(state["values"].data_ptr())
            s.numfact(_eps_magn(case))
        x = state["x"]
        x.copy_(state["b"])
        s.solve_device(x.data_ptr(), case["nrhs"], state["n"])
        if case["prec"] != "fp64":
            s.refine_device(state["b"].data_ptr(), x.data_ptr(), case["nrhs"], method)
    return x


def exact(case, seed):
    """x_true of b = A x_true, which is rounded once in 64 bits."""
    _, xt, _ = _inputs(case, seed, "cuda" if torch.cuda.is_available() else "cpu")
    return np.asfortranarray(xt.cpu().numpy().T) if case["kind"] == "host" else xt


def work(case):
    """The factorization's and the sweeps' operations; the bytes of the values, of the
    factor (written by the factorization, read by each of the two sweeps) and of the
    vectors.  Refinement is counted as one further solve (its least) with one product
    with the matrix."""
    a = _analysis(case, "cuda" if torch.cuda.is_available() else "cpu")
    st = a["st"]
    sides = 2 if case["facto"] == "getrf" else 1
    width = 8 if case["prec"] == "fp64" else 4
    factor = float(st.coefnbr) * width * sides
    vec = 8.0 * st.n * case["nrhs"]
    solves = 1 if case["prec"] == "fp64" else 2
    sweep = 4.0 * st.coefnbr * case["nrhs"]  # both sweeps
    read = factor if sides == 2 else 2 * factor
    nbytes = solves * (read + 2 * vec)
    flops = solves * sweep
    if solves == 2:
        nbytes += a["rowtab"].size * 12.0 + vec
        flops += 2.0 * a["rowtab"].size * case["nrhs"]
    if case["kind"] != "solve":
        nbytes += factor + 8.0 * a["nnz"]
        flops += st.thflops
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Largest relative error in x.  FP64 factors: rounding times the conditioning,
    2e-15 seen against x_true for the Laplacians and LU; an indefinite shift between two
    eigenvalues adds its distance to the nearest (a batch's worst of hundreds).  Refined
    solutions differ by where the iteration stops below 1e-12 in the residual: 4.6e-11
    seen, 1e-12 to 2e-9 for LDL^T over seeds, 3e-6 for the batch's worst systems."""
    if case["prec"] == "fp64":
        return {"rel": 1e-8 if _is_batch(case) else 1e-11 if case["facto"] == "sytrf" else 1e-14}
    return {"rel": 2e-5 if _is_batch(case) else 1e-8 if case["facto"] == "sytrf" else 4e-10}
