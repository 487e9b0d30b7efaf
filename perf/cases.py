"""The work that programs give this library, as cases that can be timed.

A case names a workload and its sizes. `listed()` gives the fixed ones,
`draw(rng)` more of the same ranges; `prepare` makes a case's inputs on the GPU
from a seed (and the output buffers or the plan that a program keeps), `run` is
one pass through the public entry points of nsp_b200, `work` the bytes and
operations a pass cannot do without, `exact` the same results from plain torch
in 64 bits.

Kinds of case:
  stencil   C = A*A, 7- or 27-point stencil on nx x ny x nz
  sa_ap     C = A*P, smoothed-aggregation prolongator of a 27-point stencil
  sa_rap    C = R*(A P), the second Galerkin product, R = P^T
  random    C = A*B, rectangular, row degrees uniform in [dmin, dmax]
  powerlaw  C = A*A, truncated-Pareto row degrees
  galerkin  A_c = R (A P) in one call, transpose of P included
  plan      the products of an AMG hierarchy replayed with a Plan
  batched   `count` independent random products in one call
The `api` of a product: "out" writes C into buffers that the program keeps,
"alloc" lets the library allocate C, "twocall" is the symbolic and numeric pair.
"""
from __future__ import annotations

import math
import random as _random

import torch

import nsp_b200 as nb

OMEGA = 2.0 / 3.0
DEV = "cuda"
CHUNK = 60_000_000  # intermediate products that the plain product expands at a time


def listed():
    return [
        # the smallest product of the configurations: launches and latency count
        {"name": "lap7_32", "kind": "stencil", "npts": 7, "nx": 32, "ny": 32, "nz": 32,
         "precision": "fp64", "api": "out"},
        # an ordinary Poisson operator on an odd grid, C allocated by the call
        {"name": "lap7_odd", "kind": "stencil", "npts": 7, "nx": 149, "ny": 131, "nz": 97,
         "precision": "fp64", "api": "alloc"},
        # the headline product
        {"name": "st27_128", "kind": "stencil", "npts": 27, "nx": 128, "ny": 128, "nz": 128,
         "precision": "fp64", "api": "out"},
        # the mixed-precision forms on ragged grids
        {"name": "st27_fp32c", "kind": "stencil", "npts": 27, "nx": 95, "ny": 102, "nz": 89,
         "precision": "fp32c", "api": "out"},
        {"name": "st27_fp32w_twocall", "kind": "stencil", "npts": 27, "nx": 61, "ny": 75, "nz": 83,
         "precision": "fp32w", "api": "twocall"},
        # the two products of an AMG setup's finest level
        {"name": "sa_ap_96", "kind": "sa_ap", "nx": 96, "ny": 96, "nz": 96,
         "precision": "fp64", "api": "alloc"},
        {"name": "sa_rap_96", "kind": "sa_rap", "nx": 96, "ny": 96, "nz": 96,
         "precision": "fp64", "api": "out"},
        # a whole Galerkin step of a middle level: transpose and both products
        {"name": "galerkin_50", "kind": "galerkin", "nx": 50, "ny": 47, "nz": 53},
        # an AMG re-setup with new values: the four-level hierarchy replayed
        {"name": "plan_amg_72", "kind": "plan", "nx": 72, "ny": 72, "nz": 72, "levels": 4},
        # rectangular operands without structure
        {"name": "random_rect", "kind": "random", "n": 100_003, "k": 80_021, "m": 120_011,
         "dmin": 4, "dmax": 32, "precision": "fp64", "api": "out"},
        # hub rows and load imbalance
        {"name": "powerlaw_1m", "kind": "powerlaw", "n": 1_000_000, "mean": 16.0, "maxdeg": 50_000,
         "precision": "fp64", "api": "out"},
        # many independent small and medium products
        {"name": "batched_20", "kind": "batched", "count": 20, "nmin": 1000, "nmax": 40_000,
         "dmin": 4, "dmax": 32},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["stencil", "sa_ap", "sa_rap", "galerkin", "plan", "random", "powerlaw",
                        "batched"], [6, 2, 2, 1, 1, 3, 2, 1])[0]
    prec = rng.choices(["fp64", "fp32c", "fp32w"], [4, 1, 1])[0]
    api = rng.choices(["out", "alloc", "twocall"], [4, 3, 1])[0]
    if kind == "stencil":
        while True:
            nx, ny, nz = (_logint(rng, 16, 190) for _ in range(3))
            if nx * ny * nz <= 2_000_000:
                break
        return {"kind": kind, "npts": rng.choice([7, 27, 27]), "nx": nx, "ny": ny, "nz": nz,
                "precision": prec, "api": api}
    if kind in ("sa_ap", "sa_rap"):
        nx, ny, nz = (_logint(rng, 20, 96) for _ in range(3))
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "precision": "fp64", "api": api}
    if kind == "galerkin":
        nx, ny, nz = (_logint(rng, 16, 72) for _ in range(3))
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz}
    if kind == "plan":
        nx, ny, nz = (_logint(rng, 30, 80) for _ in range(3))
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "levels": rng.choice([2, 3, 4])}
    if kind == "random":
        n, k, m = (_logint(rng, 1000, 200_000) for _ in range(3))
        dmin = rng.randint(1, 8)
        return {"kind": kind, "n": n, "k": k, "m": m, "dmin": dmin, "dmax": rng.randint(dmin + 8, 40),
                "precision": prec, "api": api}
    if kind == "powerlaw":
        n = _logint(rng, 20_000, 900_000)
        return {"kind": kind, "n": n, "mean": float(rng.randint(8, 16)), "maxdeg": max(1000, n // 20),
                "precision": prec, "api": api}
    nmax = _logint(rng, 5000, 40_000)
    return {"kind": kind, "count": rng.randint(4, 20), "nmin": 1000, "nmax": nmax, "dmin": 4,
            "dmax": rng.randint(12, 32)}


# ---- inputs: plain torch on the GPU, from the seed alone ---------------------------

class _Csr:
    """A CSR matrix in plain tensors: int32 rowptr and col, float64 val."""

    def __init__(self, nrows, ncols, rowptr, col, val):
        self.nrows, self.ncols, self.rowptr, self.col, self.val = nrows, ncols, rowptr, col, val

    def device(self, precision="fp64"):
        v = self.val if precision == "fp64" else self.val.to(torch.float32)
        return nb.DeviceCSR(self.nrows, self.ncols, self.rowptr, self.col, v)


def _gen(seed, salt):
    g = torch.Generator(device=DEV)
    g.manual_seed((int(seed) * 1_000_003 + salt) & 0x7FFFFFFFFFFF)
    return g


def _uniform(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV, dtype=torch.float64) * 2.0 - 1.0


def _rowptr(counts):
    rp = torch.zeros(counts.numel() + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(counts, 0, out=rp[1:])
    return rp.to(torch.int32)


def _stencil(nx, ny, nz, npts, seed, fp32):
    """Columns ascending; 7 points: 6 and -1; 27 points: symmetric uniform
    off-diagonals, the diagonal their absolute row sum plus one."""
    n = nx * ny * nz
    i = torch.arange(n, device=DEV)
    x, y, z = i % nx, (i // nx) % ny, i // (nx * ny)
    offs = [(dx, dy, dz) for dz in (-1, 0, 1) for dy in (-1, 0, 1) for dx in (-1, 0, 1)
            if npts == 27 or abs(dx) + abs(dy) + abs(dz) <= 1]
    p = len(offs)
    here = torch.empty(n, p, dtype=torch.bool, device=DEV)
    col = torch.empty(n, p, dtype=torch.int32, device=DEV)
    val = torch.full((n, p), -1.0, dtype=torch.float64, device=DEV)
    g = _gen(seed, 27)
    # a 7-point operator's coefficients vary a little from seed to seed
    scale = 1.0 if npts == 27 else float(_uniform(g, 1)) * 0.25 + 1.0
    for q, (dx, dy, dz) in enumerate(offs):
        here[:, q] = ((x + dx >= 0) & (x + dx < nx) & (y + dy >= 0) & (y + dy < ny)
                      & (z + dz >= 0) & (z + dz < nz))
        col[:, q] = (i + (dx + nx * (dy + ny * dz))).to(torch.int32)
    if npts == 27:
        mid = p // 2
        for q in range(mid + 1, p):
            dx, dy, dz = offs[q]
            off = dx + nx * (dy + ny * dz)
            u = _uniform(g, n)
            if fp32:
                u = u.to(torch.float32).to(torch.float64)
            val[:, q] = u
            val[:, p - 1 - q] = 0.0
            if off < n:
                val[off:, p - 1 - q] = u[:n - off]
        val[:, mid] = 0.0
        d = (val * here).abs().sum(1) + 1.0
        val[:, mid] = d.to(torch.float32).to(torch.float64) if fp32 else d
    else:
        val[:, p // 2] = 6.0
        val *= scale
        if fp32:
            val = val.to(torch.float32).to(torch.float64)
    return _Csr(n, n, _rowptr(here.sum(1)), col[here], val[here])


def _from_degrees(deg, ncols, rename, g, salt, fp32):
    """Rows of about the given degrees: uniform columns, duplicates dropped.
    The pattern comes from `salt` alone and the seed renames rows and columns
    by the permutations `rename`, so every seed has as many entries in A, B
    and C, at other places and with other values."""
    n = deg.numel()
    row = torch.repeat_interleave(torch.arange(n, device=DEV), deg.clamp(max=ncols))
    c = (torch.rand(row.numel(), generator=_gen(0, salt), device=DEV, dtype=torch.float64)
         * ncols).long()
    key = torch.unique(row * ncols + c.clamp(max=ncols - 1))
    key = torch.sort(rename[0][key // ncols] * ncols + rename[1][key % ncols])[0]
    row, col = key // ncols, (key % ncols).to(torch.int32)
    val = _uniform(g, key.numel())
    if fp32:
        val = val.to(torch.float32).to(torch.float64)
    return _Csr(n, ncols, _rowptr(torch.bincount(row, minlength=n)), col, val)


def _random_pair(n, k, m, dmin, dmax, seed, salt, fp32=False):
    """A (n x k) and B (k x m) with row degrees uniform in [dmin, dmax]."""
    g = _gen(seed, salt)
    pr, pk, pm = (torch.randperm(s, generator=g, device=DEV) for s in (n, k, m))
    dn, dk = (torch.randint(dmin, dmax + 1, (s,), generator=_gen(0, salt + 100), device=DEV)
              for s in (n, k))
    return (_from_degrees(dn, k, (pr, pk), g, salt + 200, fp32),
            _from_degrees(dk, m, (pk, pm), g, salt + 300, fp32))


def _powerlaw_csr(case, seed, fp32):
    n, mx = case["n"], case["maxdeg"]
    xmin = nb.gen.powerlaw_xmin(2.1, case["mean"], mx)
    u = torch.rand(n, generator=_gen(0, 101), device=DEV, dtype=torch.float64)
    a = 1.1
    deg = xmin * (1.0 - u * (1.0 - (xmin / mx) ** a)) ** (-1.0 / a)
    g = _gen(seed, 102)
    p = torch.randperm(n, generator=g, device=DEV)
    return _from_degrees(deg.floor().long().clamp(1, mx), n, (p, p), g, 103, fp32)


def _segments(key):
    """Distinct values of an ascending key and how often each occurs."""
    return torch.unique_consecutive(key, return_counts=True)


def _sa(A, grid):
    """P = P_tent - w D^-1 (A P_tent) for aggregates of 3 x 3 x 3 nodes."""
    nx, ny, nz = grid
    cx, cy, cz = -(-nx // 3), -(-ny // 3), -(-nz // 3)
    nc = cx * cy * cz
    i = torch.arange(A.nrows, device=DEV)
    agg = (i % nx) // 3 + cx * (((i // nx) % ny) // 3 + cy * ((i // (nx * ny)) // 3))
    row = torch.repeat_interleave(i, A.rowptr.diff().long())
    diag = torch.zeros(A.nrows, dtype=torch.float64, device=DEV)
    on = row == A.col
    diag[row[on]] = A.val[on]
    key, order = torch.sort(row * nc + agg[A.col.long()], stable=True)
    uk, cnt = _segments(key)
    s = torch.segment_reduce(A.val[order], "sum", lengths=cnt)
    r, c = uk // nc, uk % nc
    v = -OMEGA * s / diag[r]
    v = torch.where(agg[r] == c, v + 1.0, v)
    P = _Csr(A.nrows, nc, _rowptr(torch.bincount(r, minlength=A.nrows)), c.to(torch.int32), v)
    return P, (cx, cy, cz)


def _transposed(P):
    row = torch.repeat_interleave(torch.arange(P.nrows, device=DEV), P.rowptr.diff().long())
    c, order = torch.sort(P.col.long(), stable=True)
    return _Csr(P.ncols, P.nrows, _rowptr(torch.bincount(c, minlength=P.ncols)),
                row[order].to(torch.int32), P.val[order])


def _product(A, B):
    """C = A*B in 64 bits by expanding the products, sorting them by (row,
    column) and adding each entry's in A-row order; structural zeros stay."""
    blen = B.rowptr.diff().long()
    bstart = B.rowptr[:-1].long()
    ip = blen[A.col.long()]  # products of every entry of A
    pre = torch.zeros(A.nrows + 1, dtype=torch.int64, device=DEV)
    tot = torch.zeros(ip.numel() + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(ip, 0, out=tot[1:])
    pre = tot[A.rowptr.long()]
    cuts, r0, host = [0], 0, pre.cpu()
    while r0 < A.nrows:
        r1 = int(torch.searchsorted(host, int(host[r0]) + CHUNK, right=True)) - 1
        r0 = min(max(r1, r0 + 1), A.nrows)
        cuts.append(r0)
    keys, vals = [], []
    arow = torch.repeat_interleave(torch.arange(A.nrows, device=DEV), A.rowptr.diff().long())
    for r0, r1 in zip(cuts, cuts[1:]):
        e0, e1 = int(A.rowptr[r0]), int(A.rowptr[r1])
        n = ip[e0:e1]
        rep = torch.repeat_interleave(torch.arange(e0, e1, device=DEV), n)
        within = torch.arange(rep.numel(), device=DEV) - (tot[rep] - tot[e0])
        b = bstart[A.col.long()[rep]] + within
        key, order = torch.sort(arow[rep] * B.ncols + B.col.long()[b], stable=True)
        v = (A.val[rep] * B.val[b])[order]
        uk, cnt = _segments(key)
        keys.append(uk)
        vals.append(torch.segment_reduce(v, "sum", lengths=cnt) if cnt.numel() else v)
        del rep, within, b, key, order, v
    key = torch.cat(keys) if keys else torch.zeros(0, dtype=torch.int64, device=DEV)
    val = torch.cat(vals) if vals else torch.zeros(0, dtype=torch.float64, device=DEV)
    row = key // B.ncols
    return _Csr(A.nrows, B.ncols, _rowptr(torch.bincount(row, minlength=A.nrows)),
                (key % B.ncols).to(torch.int32), val)


def _hierarchy(case, seed):
    """The pairs (A_l, P_l), (R_l, A_l P_l) of the case's levels."""
    grid = (case["nx"], case["ny"], case["nz"])
    A = _stencil(*grid, 27, seed, False)
    pairs = []
    for _ in range(case["levels"] - 1):
        P, grid = _sa(A, grid)
        R = _transposed(P)
        AP = _product(A, P)
        pairs += [(A, P), (R, AP)]
        A = _product(R, AP)
    return pairs


def _batch(case, seed):
    r = _random.Random(case["count"])
    pairs = []
    for p in range(case["count"]):
        n = r.randint(case["nmin"], case["nmax"])
        pairs.append(_random_pair(n, n, n, case["dmin"], case["dmax"], seed, 1000 * (p + 1)))
    return pairs


def _operands(case, seed):
    """The pairs (A, B) whose products the case forms."""
    kind, fp32 = case["kind"], case.get("precision", "fp64") != "fp64"
    if kind == "stencil":
        A = _stencil(case["nx"], case["ny"], case["nz"], case["npts"], seed, fp32)
        return [(A, A)]
    if kind in ("sa_ap", "sa_rap", "galerkin"):
        grid = (case["nx"], case["ny"], case["nz"])
        A = _stencil(*grid, 27, seed, False)
        P, _ = _sa(A, grid)
        return [(_transposed(P), _product(A, P))] if kind == "sa_rap" else [(A, P)]
    if kind == "random":
        return [_random_pair(case["n"], case["k"], case["m"], case["dmin"], case["dmax"], seed, 1,
                             fp32)]
    if kind == "powerlaw":
        A = _powerlaw_csr(case, seed, fp32)
        return [(A, A)]
    return _hierarchy(case, seed) if kind == "plan" else _batch(case, seed)


def prepare(case, seed):
    pairs = _operands(case, seed)
    prec = case.get("precision", "fp64")
    dev = {}

    def put(M):
        if id(M) not in dev:
            dev[id(M)] = M.device(prec)
        return dev[id(M)]
    As, Bs = [put(a) for a, _ in pairs], [put(b) for _, b in pairs]
    state = {"case": dict(case), "A": As, "B": Bs}
    if case.get("api") == "out":  # C's buffers, sized once and kept
        rp, nnz = nb.spgemm_symbolic(As[0], Bs[0])
        state["out"] = nb.DeviceCSR(As[0].nrows, Bs[0].ncols, rp,
                                    torch.empty(max(nnz, 1), dtype=torch.int32, device=DEV),
                                    torch.empty(max(nnz, 1), dtype=torch.float64, device=DEV))
    if case["kind"] == "plan":
        state["plan"] = nb.Plan(As, Bs, check_errors=False)
    torch.cuda.synchronize()
    return state


def _outputs(C):
    return {"rowptr": C.rowptr, "col": C.col, "val": C.val}


def run(state):
    case, As, Bs = state["case"], state["A"], state["B"]
    kind = case["kind"]
    if kind == "plan":
        state["plan"].execute()
        return [_outputs(C) for C in state["plan"].C]
    if kind == "batched":
        return [_outputs(C) for C in nb.spgemm_batched(As, Bs)]
    if kind == "galerkin":
        Ac, R = nb.galerkin(As[0], Bs[0], return_R=True)
        return [_outputs(Ac), _outputs(R)]
    prec, api = case["precision"], case["api"]
    if api == "twocall":
        rp, nnz = nb.spgemm_symbolic(As[0], Bs[0])
        return _outputs(nb.spgemm_numeric(As[0], Bs[0], rp, nnz, precision=prec))
    return _outputs(nb.spgemm(As[0], Bs[0], precision=prec, out=state.get("out")))


# ---- what a pass cannot do without -------------------------------------------------

def _line(n, reach):
    """Entries of a 1-D band of half width `reach` on n nodes."""
    return sum(min(i + reach, n - 1) - max(i - reach, 0) + 1 for i in range(n))


def _sa_line(n):
    """1-D counts of the smoothed aggregation on n nodes: entries of P, A P and
    R (A P), and the products of A*P and of R*(A P)."""
    a = [(max(i - 1, 0), min(i + 1, n - 1)) for i in range(n)]
    p = [(lo // 3, hi // 3) for lo, hi in a]
    ap = [(p[lo][0], p[hi][1]) for lo, hi in a]
    nc = -(-n // 3)
    r = [[] for _ in range(nc)]
    for i, (lo, hi) in enumerate(p):
        for c in range(lo, hi + 1):
            r[c].append(i)
    size = lambda s: s[1] - s[0] + 1  # noqa: E731
    return {"p": sum(map(size, p)), "ap": sum(map(size, ap)),
            "rap": sum(max(ap[i][1] for i in s) - min(ap[i][0] for i in s) + 1 for s in r),
            "ip_ap": sum(size(p[j]) for lo, hi in a for j in range(lo, hi + 1)),
            "ip_rap": sum(size(ap[i]) for s in r for i in s)}


def _cube(f, dims):
    return math.prod(f(d) for d in dims)


def _csr_bytes(nrows, nnz, w=8):
    return 4 * (nrows + 1) + (4 + w) * nnz


def _counts(case):
    """[(rows and entries of A, of B, of C, intermediate products)] of the
    case's products; expected values where the inputs are random."""
    kind = case["kind"]
    if kind == "stencil":
        d = (case["nx"], case["ny"], case["nz"])
        n = math.prod(d)
        if case["npts"] == 27:
            a, c = _cube(lambda k: _line(k, 1), d), _cube(lambda k: _line(k, 2), d)
            ip = _cube(lambda k: 9 * k - 10 if k > 1 else 1, d)
            return [((n, a), (n, a), (n, c), ip)]
        m = sum(n // k * 2 * (k - 1) for k in d)  # off-diagonal entries
        two = sum(n // k * 2 * (k - 2) for k in d)
        mixed = sum(2 * 4 * (d[i] - 1) * (d[j] - 1) * (n // (d[i] * d[j]))
                    for i in range(3) for j in range(i)) // 2
        ip = sum(n // k * (4 * (k - 2) + 2) for k in d) + 2 * m + n + 2 * mixed
        return [((n, n + m), (n, n + m), (n, n + m + two + mixed), ip)]
    if kind in ("sa_ap", "sa_rap", "galerkin", "plan"):
        d, got = (case["nx"], case["ny"], case["nz"]), []
        for _ in range(case.get("levels", 2) - 1):
            n, a = math.prod(d), _cube(lambda k: _line(k, 1), d)
            s = {w: _cube(lambda k: _sa_line(k)[w], d) for w in ("p", "ap", "rap", "ip_ap", "ip_rap")}
            d = tuple(-(-k // 3) for k in d)
            nc = math.prod(d)
            got += [((n, a), (n, s["p"]), (n, s["ap"]), s["ip_ap"]),
                    ((nc, s["p"]), (n, s["ap"]), (nc, s["rap"]), s["ip_rap"])]
        return got[:1] if kind == "sa_ap" else got[1:] if kind == "sa_rap" else got
    if kind == "random":
        n, k, m, deg = case["n"], case["k"], case["m"], (case["dmin"] + case["dmax"]) / 2
        c = m * -math.expm1(-deg * deg / m)
        return [((n, n * deg), (k, k * deg), (n, n * c), n * deg * deg)]
    if kind == "powerlaw":
        n, deg = case["n"], case["mean"]
        return [((n, n * deg), (n, n * deg), (n, n * deg * deg), n * deg * deg)]
    n, deg = (case["nmin"] + case["nmax"]) / 2, (case["dmin"] + case["dmax"]) / 2
    return [((n, n * deg), (n, n * deg), (n, n * deg * deg), n * deg * deg)] * case["count"]


def work(case):
    w = 8 if case.get("precision", "fp64") == "fp64" else 4
    nbytes = flops = 0.0
    for a, b, c, ip in _counts(case):
        nbytes += _csr_bytes(*a, w) + _csr_bytes(*b, w) + _csr_bytes(*c)
        flops += 2.0 * ip
    if case["kind"] == "galerkin":  # A and P read once, R and A_c written once
        (a, p, _, _), (r, _, c, _) = _counts(case)
        nbytes = _csr_bytes(*a) + _csr_bytes(*p) + _csr_bytes(*r) + _csr_bytes(*c)
    return {"bytes": float(nbytes), "flops": float(flops)}


# ---- the same results in 64 bits without the library -------------------------------

def exact(case, seed):
    pairs = _operands(case, seed)
    kind = case["kind"]

    def values(M):
        return {"rowptr": None, "col": None, "val": M.val}
    if kind == "galerkin":
        (A, P), = pairs
        R = _transposed(P)
        return [values(_product(R, _product(A, P))), values(R)]
    got = [values(_product(A, B)) for A, B in pairs]
    return got if kind in ("plan", "batched") else got[0]
