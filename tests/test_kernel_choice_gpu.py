"""Which kernels a product takes, on both sides of the lines: lists or hash kernels by
products an entry, a two-call numeric step whose A reads B's long rows above all, and rows
of more products than runs hold. Values against the oracle; the search for runs by the
launches of a call that is told to search (row_kernel 8)."""
import numpy as np
import pytest

import nsp_b200 as nb
import oracle
from nsp_b200.csr import HostCSR

from conftest import assert_bitwise, assert_same_structure
from test_run_search_gpu import RUNS, launches

pytestmark = pytest.mark.gpu


def check(A, B, precision="fp64"):
    f = lambda h: HostCSR(h.nrows, h.ncols, h.rowptr, h.col, h.val.astype(np.float32))  # noqa: E731
    dA, dB = (A, B) if precision == "fp64" else (f(A), f(B))
    dA, dB = dA.to_device(), dB.to_device()
    rp, col, val = oracle.spgemm(A, B)
    bound = oracle.absbound(A, B, rp, col)
    one, st = nb.spgemm(dA, dB, precision=precision, return_stats=True)
    rp2, nnz = nb.spgemm_symbolic(dA, dB)
    two = nb.spgemm_numeric(dA, dB, rp2, nnz, precision=precision)
    short = np.repeat(np.diff(rp) <= 512, np.diff(rp))
    tol = 1e-10 if precision == "fp32c" else 2 * int(np.diff(A.rowptr).max()) * 2.0**-53
    for C in (one, two):
        C = C.to_host()
        assert_same_structure(C.rowptr, C.col, rp, col)
        assert np.all(np.abs(C.val - val) <= tol * bound)
        if precision != "fp32c":
            assert_bitwise(C.val[short], val[short])
    return st


def values(h):
    h.val[:] = h.val.astype(np.float32)
    return h


# d * d products a row over m columns
@pytest.mark.parametrize("precision", ["fp64", "fp32w", "fp32c"])
@pytest.mark.parametrize("x", [0.40, 0.46, 0.54, 0.70, 0.85])  # 1.21 to 1.48 products an entry
@pytest.mark.parametrize("d", [4, 16, 24, 34])
def test_products_an_entry(cuda, d, x, precision):
    m = int(d * d / x)
    A = values(nb.gen.random(700, 900, d, d, seed=1))
    B = values(nb.gen.random(900, max(m, d), d, d, seed=2))
    st = check(A, B, precision)
    assert 1.1 < st["intprod"] / st["nnz"] < 1.6


@pytest.mark.parametrize("per_row", [1, 10, 40])
@pytest.mark.parametrize("n", [900, 5000, 20_000])
def test_a_reads_the_long_rows(cuda, n, per_row):
    """400 B rows of 60 entries of 600 columns among 20,000 of one entry."""
    rng = np.random.default_rng(n + per_row)
    k, hub, m = 20_000, 400, 5000
    rows = [np.sort(rng.choice(600, 60, replace=False)) for _ in range(hub)]
    rows += [rng.integers(0, m, 1) for _ in range(k - hub)]
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    B = HostCSR(k, m, rp, np.concatenate(rows).astype(np.int32), rng.uniform(-1, 1, rp[-1]))
    col = np.concatenate([np.sort(rng.choice(hub, per_row, replace=False)) for _ in range(n)])
    A = HostCSR(n, k, np.arange(0, n * per_row + 1, per_row, dtype=np.int32), col.astype(np.int32),
                rng.uniform(-1, 1, n * per_row))
    check(A, B)


def unknowns(H, d, rng):
    """A grid of d unknowns a node."""
    r, c = np.repeat(np.arange(H.nrows), np.diff(H.rowptr)), H.col.astype(np.int64)
    a = np.arange(d)
    cols = (c[:, None] * d + a).reshape(-1)  # one row of each node
    lens = np.repeat(np.diff(H.rowptr) * d, d)
    starts = H.rowptr[:-1] * d
    col = np.concatenate([cols[s:s + n] for s, n in zip(np.repeat(starts, d), lens)])
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    return HostCSR(H.nrows * d, H.ncols * d, rp, col.astype(np.int32), rng.uniform(-1, 1, rp[-1]))


def test_rows_of_too_many_products(cuda):
    """27-point grid of 3 unknowns a node: rows of 81 entries and 6561 products."""
    X = unknowns(nb.gen.stencil(14, npts=27), 3, np.random.default_rng(1))
    d = X.to_device()
    for two in (False, True):
        auto, told = launches(d, d, 0, two), launches(d, d, RUNS, two)
        assert all(x != y for x, y in zip(auto, told)), (auto, told)
    check(X, X)
