"""The rules that send rows to the row-run kernels, restated in numpy: the
column shifts of B's rows, the link codes of A's rows, the runs, and the layout
of a tile (segments of B staged in shared memory, the place and stride of every
product). For every run found: each row's products land on the first row's
entries moved by one shift, and the staged place of every product of every row
of every tile holds exactly the value the plain product reads, inside the
staged area. Inputs: stencils, aggregation products, block and band matrices,
and those with columns moved, rows emptied, rows unsorted or repeated."""
import numpy as np
import pytest

import nsp_b200 as nb
from nsp_b200.csr import HostCSR

NO, ANY = None, "any"
MAX_LAG, MAX_LEN, MAX_A, MAX_IP, RUN_MIN, BLOCK = 3, 128, 128, 1536, 6, 512
SMALL_IP, REACH = 256, 512
CLASS = {False: (50 * 1024, 8), True: (110000, 16)}  # shared memory, warps


def shifts(B):
    rp, col = B.rowptr, B.col
    out = [[NO] * B.nrows for _ in range(MAX_LAG + 1)]
    for k in range(B.nrows):
        ln = rp[k + 1] - rp[k]
        for g in range(1, MAX_LAG + 1):
            if k < g or ln > MAX_LEN or rp[k - g + 1] - rp[k - g] != ln:
                continue
            if g > 1 and (k < 2 * g or rp[k] - rp[k - g] != rp[k - g] - rp[k - 2 * g]):
                continue
            d = col[rp[k]:rp[k + 1]].astype(np.int64) - col[rp[k - g]:rp[k - g] + ln]
            if ln == 0:
                out[g][k] = ANY
            elif (d == d[0]).all():
                out[g][k] = int(d[0])
    return out


def codes(A, B, bdel, lags):
    rp, col, blen = A.rowptr, A.col, np.diff(B.rowptr)
    out = np.zeros(A.nrows, np.int32)
    for i in range(A.nrows):
        a = col[rp[i]:rp[i + 1]]
        ip = int(blen[a].sum())
        if not (0 < len(a) <= MAX_A and 0 < ip <= MAX_IP):
            continue
        for s in range(1, min(MAX_LAG, i) + 1):
            p = col[rp[i - s]:rp[i - s + 1]]
            if len(p) != len(a):
                continue
            sigma = int(a[0]) - int(p[0])
            if not 1 <= sigma <= MAX_LAG or sigma not in lags or (a - p != sigma).any():
                continue
            if A is B and bdel[s][i] != sigma:  # taken from the shifts (stricter past lag 1)
                continue
            d = [bdel[sigma][k] for k in a]
            if NO in d or len({x for x in d if x != ANY}) != 1:
                continue
            if not out[i] or sigma == s:
                out[i] = s | sigma << 2
            if sigma == s:
                break
    return out


def runs_of(code):
    found = []
    for b0 in range(0, len(code), BLOCK):
        c = code[b0:b0 + BLOCK]
        for t in range(len(c)):
            s = c[t] & 3
            if not c[t] or (t >= s and c[t - s] == c[t]):
                continue
            rows = list(range(t, len(c), s))
            rows = rows[:next((q for q, j in enumerate(rows) if c[j] != c[t]), len(rows))]
            if t >= s and c[t - s] == 0 and all((c[t - s + g] & 3) != g for g in range(1, s)):
                rows.insert(0, t - s)
            if len(rows) >= RUN_MIN:
                found.append(([b0 + r for r in rows], int(s), int(c[t] >> 2)))
    return found


def tile_rows(A, B, rows, sigma, vsz):
    """Rows, places and segments of a program's tiles, as the kernel lays them out."""
    rp = B.rowptr.astype(np.int64)
    ks = A.col[A.rowptr[rows[0]]:A.rowptr[rows[0] + 1]].astype(np.int64)
    na, n_len = len(ks), rp[ks + 1] - rp[ks]
    P, pl = int(n_len.sum()), rp[ks + sigma] - rp[ks]
    n = len(np.unique(np.concatenate([B.col[rp[k]:rp[k + 1]] for k in ks])))
    smem, warps = CLASS[P > SMALL_IP]

    def near(t):
        return ks[t] >= ks[t - 1] and ks[t] - ks[t - 1] <= REACH and pl[t] == pl[t - 1]

    unit = 16 // vsz  # values between two 16-byte boundaries

    def layout(L):
        off, seg, x = np.zeros(na, np.int64), [], 0
        for t in range(na):
            if t == 0 or not near(t) or ks[t] - ks[t - 1] >= (L - 1) * sigma + 1:
                x += rp[ks[t]] - (0 if t == 0 else rp[ks[t - 1]] + (L - 1) * pl[t - 1] + n_len[t - 1])
                seg.append([t, t])
            seg[-1][1] = t
            off[t] = rp[ks[t]] - x + 3 * unit * (len(seg) - 1)
        return off, seg, int(off[-1] + (L - 1) * pl[-1] + n_len[-1] + 3 * unit)

    def fits(L):
        up = lambda v: (v + 15) & ~15  # noqa: E731
        fixed = (up(8 * (P + 32) + 4 * n) + up(L * (n | 1) * 8 + 16) + L * up(na * vsz + 16) + 16)
        return fixed + layout(L)[2] * vsz <= smem
    assert fits(1)
    lo, hi = 1, 128 + 1
    while hi - lo > 1:
        mid = (lo + hi) // 2
        lo, hi = (mid, hi) if fits(mid) else (lo, mid)
    L = lo & ~31 if lo > 32 else lo
    off, seg, total = layout(L)
    # places count from the segments' 16-byte boundaries; a word holds their bytes
    # in 17 bits and the rows' distance in 15
    place, segs = np.zeros(na, np.int64), []
    for t0, t1 in seg:
        dst = off[t0] & ~(unit - 1)
        place[t0:t1 + 1] = off[t0:t1 + 1] - off[t0] + dst
        segs.append((t0, t1, dst))
    assert warps // -(-L // 32) >= 1 and total * vsz < 1 << 17 and (L == 1 or (pl < 1 << 15).all())
    return L, place, segs, total, pl, n_len


def check(A, B, vsz=8):
    bdel = shifts(B)
    lags = {g for g in range(1, MAX_LAG + 1)
            if 5 * sum(x is not NO for x in bdel[g]) >= 2 * B.nrows}
    code = codes(A, B, bdel, lags)
    runs = runs_of(code)
    rp, used = B.rowptr, np.zeros(A.nrows, int)
    for rows, s, sigma in runs:
        used[rows] += 1
        first = None
        for r in rows:
            ks = A.col[A.rowptr[r]:A.rowptr[r + 1]]
            pat = ([int(rp[k + 1] - rp[k]) for k in ks],
                   np.concatenate([B.col[rp[k]:rp[k + 1]] for k in ks]).astype(np.int64))
            if first is None:
                first = pat
            assert pat[0] == first[0]
            assert len(set((pat[1] - first[1]).tolist())) == 1
        L, place, segs, total, pl, n_len = tile_rows(A, B, rows, sigma, vsz)
        unit = 16 // vsz
        ks = A.col[A.rowptr[rows[0]]:A.rowptr[rows[0] + 1]].astype(np.int64)
        for j in range(0, len(rows), L):
            cnt = min(L, len(rows) - j)
            staged = np.full(total, -1, np.int64)  # which entry of B each place holds
            lead = np.zeros(len(place), np.int64)
            for t0, t1, dst in segs:
                b0, b1 = rp[ks[t0] + sigma * j], rp[ks[t1] + sigma * (j + cnt - 1) + 1]
                lead[t0:t1 + 1] = b0 % unit  # values before it on its boundary
                c0, c1 = b0 - b0 % unit, -(-b1 // unit) * unit
                assert dst >= 0 and dst % unit == 0 and dst + c1 - c0 <= total
                assert (staged[dst:dst + c1 - c0] == -1).all()  # copies never overlap
                staged[dst:dst + c1 - c0] = np.arange(c0, c1)
            for l in range(cnt):
                r = rows[j + l]
                for t, k in enumerate(A.col[A.rowptr[r]:A.rowptr[r + 1]]):
                    at = place[t] + lead[t] + np.arange(n_len[t]) + pl[t] * l
                    assert (at < total).all()
                    assert np.array_equal(staged[at], np.arange(rp[k], rp[k] + n_len[t]))
    assert used.max(initial=0) <= 1
    return runs, used


def csr(rows, ncols, rng):
    rp = np.zeros(len(rows) + 1, np.int32)
    rp[1:] = np.cumsum([len(r) for r in rows])
    col = np.concatenate([np.asarray(r, np.int32) for r in rows]) if rp[-1] else np.zeros(0, np.int32)
    return HostCSR(len(rows), ncols, rp, col.astype(np.int32), rng.uniform(-1, 1, rp[-1]))


def rows_of(M):
    return [M.col[M.rowptr[i]:M.rowptr[i + 1]].tolist() for i in range(M.nrows)]


def prolongator(nx, ny, nz, agg=3):
    """Pattern of the smoothed prolongator of an agg^3 aggregation, and of its
    transpose and the product A*P."""
    import scipy.sparse as sp
    A = nb.gen.stencil(nx, ny, nz, npts=27)
    c = [-(-d // agg) for d in (nx, ny, nz)]
    i = np.arange(nx * ny * nz)
    g = i % nx // agg + c[0] * (i // nx % ny // agg + c[1] * (i // (nx * ny) // agg))
    T = sp.csr_matrix((np.ones(len(i)), (i, g)), shape=(len(i), c[0] * c[1] * c[2]))
    S = sp.csr_matrix((np.ones(A.nnz), A.col, A.rowptr), shape=(A.nrows, A.nrows))
    P = (S @ T).tocsr()
    out = []
    for M in (P, P.T.tocsr(), (S @ P).tocsr()):
        M.sort_indices()
        out.append(HostCSR(M.shape[0], M.shape[1], M.indptr.astype(np.int32),
                           M.indices.astype(np.int32), np.ones(M.nnz)))
    return A, *out


@pytest.mark.parametrize("npts,dims", [(27, (40, 6, 5)), (7, (35, 9, 6)), (7, (200, 4, 3)),
                                       (27, (13, 7, 7)), (27, (1, 30, 30))])
@pytest.mark.parametrize("vsz", [4, 8])
def test_stencils(npts, dims, vsz):
    A = nb.gen.stencil(*dims, npts=npts)
    runs, used = check(A, A, vsz)
    if dims[0] >= 35:  # most interior rows; runs also end every 512 rows
        assert used.mean() > 0.8


@pytest.mark.parametrize("agg", [2, 3])
def test_aggregation_products(agg):
    A, P, R, AP = prolongator(45, 7, 8, agg)
    runs, used = check(A, P)
    assert used.mean() > 0.5 and all(s == agg and sg == agg for _, s, sg in runs)
    runs, used = check(R, AP)
    assert used.mean() > 0.4 and all(s == 1 and sg == agg for _, s, sg in runs)


def test_several_unknowns_a_node():
    rng = np.random.default_rng(2)
    base = rows_of(nb.gen.stencil(30, 3, 3, npts=7))
    for d in (2, 3):  # d x d blocks on a 7-point pattern
        A = csr([[d * c + u for c in r for u in range(d)] for r in base for _ in range(d)],
                d * len(base), rng)
        _, used = check(A, A)
        assert used.mean() > 0.5


def test_band_and_repeated_columns():
    rng = np.random.default_rng(3)
    n = 700
    band = csr([[c for c in (i - 9, i - 1, i, i + 1, i + 9) if 0 <= c < n] for i in range(n)], n, rng)
    _, used = check(band, band)
    assert used.mean() > 0.9
    # A rows out of order, with a column twice; B rows out of order
    odd = csr([[c for c in (i + 9, i, i - 1, i, i + 2) if 0 <= c < n] for i in range(n)], n, rng)
    _, used = check(odd, band)
    assert used.mean() > 0.9
    check(odd, odd)
    # rows of one entry, and B rows that are empty for whole stretches
    one = csr([[i] for i in range(n)], n, rng)
    holes = csr([r if i % 90 < 70 else [] for i, r in enumerate(rows_of(band))], n, rng)
    check(one, holes)
    check(band, holes)


@pytest.mark.parametrize("seed", range(6))
def test_almost_structured(seed):
    """Stencil and aggregation patterns with columns moved, rows emptied or
    swapped: every run that is still found must hold."""
    rng = np.random.default_rng(seed)
    A, P, R, AP = prolongator(24, 5, 5)

    def spoil(M, frac):
        rows = rows_of(M)
        for i in rng.choice(M.nrows, max(1, int(frac * M.nrows)), replace=False):
            how = rng.integers(4)
            if how == 0 and rows[i]:
                rows[i][rng.integers(len(rows[i]))] = int(rng.integers(M.ncols))
                rows[i] = sorted(set(rows[i]))
            elif how == 1:
                rows[i] = []
            elif how == 2:
                j = int(rng.integers(M.nrows))
                rows[i], rows[j] = rows[j], rows[i]
            else:
                rows[i] = [min(c + 1, M.ncols - 1) for c in rows[i]]
        return csr(rows, M.ncols, rng)
    for X, Y in ((A, A), (A, P), (R, AP)):
        f = 0.02 if seed % 2 else 0.1
        check(spoil(X, f), Y)
        check(X, spoil(Y, f))
        Z = spoil(X, f)
        check(Z, spoil(Y, f) if X is not Y else Z)


def test_unstructured_has_no_runs():
    A = nb.gen.random(600, 600, 3, 9, seed=4)
    assert not check(A, A)[0]
