"""Row runs (k_brow_delta, k_run_list, k_num_run): rows that repeat a pattern at
a fixed distance are counted once a run and computed by one program a run.
Values are sums in A-row order from zero, like the oracle's, so they are
compared bit for bit; with runs off (opts.row_kernel bit 0x10000) the bytes
must be the same. Sizes: runs shorter and longer than a row group of 32 lanes,
tiles of several row groups, partial last tiles, runs cut at 512 rows, one and
several programs a block, both value types, every entry point with runs."""
import numpy as np
import pytest

import nsp_b200 as nb
import oracle
from nsp_b200 import amg
from nsp_b200.csr import HostCSR

from conftest import assert_bitwise, assert_same_structure
from test_row_run_cpu import csr, prolongator, rows_of

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def runs_at_any_size(monkeypatch):
    # opts.row_kernel 8: runs for these small products too
    monkeypatch.setenv("NSPB_ROW_KERNEL", "8")

NO_RUNS = 0x10000


def as32(h):
    return HostCSR(h.nrows, h.ncols, h.rowptr, h.col, h.val.astype(np.float32))


def rounded(h):
    return HostCSR(h.nrows, h.ncols, h.rowptr, h.col, h.val.astype(np.float32).astype(np.float64))


def with_values(h, seed):
    v = np.random.default_rng(seed).uniform(-1, 1, h.nnz)
    return HostCSR(h.nrows, h.ncols, h.rowptr, h.col, v)


def check(A, B, precision="fp64"):
    X, Y = (A, B) if precision == "fp64" else (as32(A), as32(B))
    dA = X.to_device()
    dB = dA if A is B else Y.to_device()
    C = nb.spgemm(dA, dB, precision=precision)
    rp, nnz = nb.spgemm_symbolic(dA, dB)
    C2 = nb.spgemm_numeric(dA, dB, rp, nnz, precision=precision).to_host()
    off = nb.spgemm(dA, dB, precision=precision, row_kernel=NO_RUNS).to_host()
    got = C.to_host()
    W = (A, B) if precision == "fp64" else (rounded(A), rounded(B))
    rp, col, val = oracle.spgemm(*W)
    for c in (got, C2, off):
        assert_same_structure(c.rowptr, c.col, rp, col)
    if precision == "fp32c":  # the mode's bound (the numeric call asks for 1e-12: fp64 rows)
        bound = oracle.absbound(*W, rp, col)
        assert np.all(np.abs(got.val - val) <= 1e-10 * bound)
        assert np.all(np.abs(C2.val - val) <= 1e-12 * bound)
        assert_bitwise(off.val, got.val)  # the same pairs in the same order
    else:
        assert_bitwise(got.val, val)
        assert_bitwise(C2.val, val)


@pytest.mark.parametrize("dims", [(40, 9, 7), (131, 5, 6), (33, 34, 3), (10, 10, 10), (520, 4, 3)])
@pytest.mark.parametrize("npts", [7, 27])
@pytest.mark.parametrize("precision", ["fp64", "fp32c", "fp32w"])
def test_stencils(cuda, dims, npts, precision):
    A = nb.gen.stencil(*dims, npts=npts, fp32=precision != "fp64")
    check(A, A, precision)


@pytest.mark.parametrize("agg", [2, 3])
@pytest.mark.parametrize("precision", ["fp64", "fp32w"])
def test_aggregation_products(cuda, agg, precision):
    A, P, R, AP = prolongator(62, 17, 16, agg)
    for q, (X, Y) in enumerate(((A, P), (R, AP))):
        X, Y = (with_values(M, 5 + q) for M in (X, Y))
        if precision != "fp64":
            X, Y = rounded(X), rounded(Y)
        check(X, Y, precision)


def test_bands_blocks_and_odd_rows(cuda):
    rng = np.random.default_rng(7)
    n = 3000
    band = csr([[c for c in (i - 9, i - 1, i, i + 1, i + 9) if 0 <= c < n] for i in range(n)], n, rng)
    check(band, band)
    # A rows out of order with a repeated column, over sorted B rows
    odd = csr([[c for c in (i + 9, i, i - 1, i, i + 2) if 0 <= c < n] for i in range(n)], n, rng)
    check(odd, band)
    one = csr([[i] for i in range(n)], n, rng)
    check(one, band)
    holes = csr([r if i % 90 < 70 else [] for i, r in enumerate(rows_of(band))], n, rng)
    check(band, holes)
    base = rows_of(nb.gen.stencil(60, 5, 5, npts=7))
    for d in (2, 3):
        M = csr([[d * c + u for c in r for u in range(d)] for r in base for _ in range(d)],
                d * len(base), rng)
        check(M, M)


def test_long_patterns(cuda):
    # rows of up to 1536 products: tiles of a few rows, large programs
    rng = np.random.default_rng(8)
    n = 1500
    for reach in (9, 14, 18, 19, 20):  # 37^2 = 1369 products a row, then past 1536
        M = csr([list(range(max(0, i - reach), min(n, i + reach + 1))) for i in range(n)], n, rng)
        check(M, M)
    # far-apart entries: no segment of B shared between two entries of A
    far = csr([[c for c in (i - 400, i - 200, i, i + 200, i + 400) if 0 <= c < n] for i in range(n)],
              n, rng)
    check(far, far)


@pytest.mark.parametrize("frac", [0.003, 0.05])
def test_moved_columns(cuda, frac):
    from test_row_template_gpu import perturb
    A = nb.gen.stencil(50, 12, 11, npts=27)
    P = perturb(A, frac, seed=3)
    check(P, A)
    check(A, P)
    check(P, P)


def test_plan_and_batch(cuda):
    pairs = amg.amg_batch(L=27, levels=3)
    A = nb.gen.stencil(45, 8, 9, npts=27)
    pairs += [(A, A), (nb.gen.random(500, 400, 1, 9, seed=1), nb.gen.random(400, 300, 1, 9, seed=2))]
    dA, dB = [a.to_device() for a, _ in pairs], [b.to_device() for _, b in pairs]
    want = [oracle.spgemm(a, b) for a, b in pairs]
    for C, (rp, col, val) in zip(nb.spgemm_batched(dA, dB), want):
        h = C.to_host()
        assert_same_structure(h.rowptr, h.col, rp, col)
        assert_bitwise(h.val, val)
    for group in (0, 1):  # all products in one table; one product a group
        plan = nb.Plan(dA, dB, max_group=group)
        for a in dA:
            a.val.mul_(-2.0)
        plan.execute()
        for C, (rp, col, val) in zip(plan.C, want):
            h = C.to_host()
            assert_same_structure(h.rowptr, h.col, rp, col)
            assert_bitwise(h.val, -2.0 * val)
        for a in dA:
            a.val.mul_(-0.5)


def test_special_values(cuda):
    A = nb.gen.stencil(40, 6, 5, npts=27)
    v = A.val.copy()
    v[::97], v[5::89], v[7::83], v[11::3] = np.inf, -np.inf, np.nan, -0.0
    A = HostCSR(A.nrows, A.ncols, A.rowptr, A.col, v)
    dA = A.to_device()
    got = nb.spgemm(dA, dA).to_host()
    off = nb.spgemm(dA, dA, row_kernel=NO_RUNS).to_host()
    assert np.array_equal(got.val, off.val, equal_nan=True)
    fin = ~np.isnan(got.val)
    assert np.array_equal(np.signbit(got.val[fin]), np.signbit(off.val[fin]))


def test_counts_and_pairs_reported(cuda):
    A = nb.gen.stencil(45, 9, 8, npts=27, fp32=True)
    d = as32(A).to_device()
    on, s1 = nb.spgemm(d, d, precision="fp32c", return_stats=True)
    off, s0 = nb.spgemm(d, d, precision="fp32c", row_kernel=NO_RUNS, return_stats=True)
    for k in ("intprod", "nnz", "sym_bins", "num_bins", "rows_redone", "max_row_err", "b_sorted"):
        assert s1[k] == s0[k], k
    assert_bitwise(on.to_host().val, off.to_host().val)  # the same pairs in the same order
    _, s = nb.spgemm(d, d, precision="fp32c", comp_tol=1e-15, return_stats=True)
    assert s["rows_redone"] == A.nrows
