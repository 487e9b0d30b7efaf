"""Rows of C that are one row of B, scaled (a diagonal or a permutation times B): rows in
order are taken as they are, others sorted, in the same kernel."""
import numpy as np
import pytest

import nsp_b200 as nb
import oracle
from nsp_b200.csr import HostCSR

from conftest import assert_bitwise, assert_same_structure

pytestmark = pytest.mark.gpu

M = 5003
LENS = [0, 1, 2, 16, 17, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 160, 161, 300]


def b_rows(rng, kind):
    lens = np.tile(LENS, 30)
    cols = []
    for i, d in enumerate(lens):
        if kind == "crowded":  # side by side, as the rows of a stencil
            c = int(rng.integers(0, M - 400)) + np.arange(d)
        else:
            c = np.sort(rng.choice(M, d, replace=False))
        if kind == "any order" and d > 1 and i % 3:
            if i % 3 == 1:
                c[-2:] = c[-2:][::-1]  # the last two only
            else:
                c = rng.permutation(c)
        cols.append(c)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    val = rng.uniform(-1, 1, rp[-1]).astype(np.float32).astype(np.float64)
    val[::11] = 0.0
    return HostCSR(len(lens), M, rp, np.concatenate(cols).astype(np.int32), val)


def a_rows(rng, k, kind, empty):
    """One entry a row; or also entries of empty B rows around it; or a few rows of more."""
    rows = [[i] for i in rng.permutation(k)]
    if kind == "empty rows too":
        rows = [sorted({*r, *rng.choice(empty, 2)}) for r in rows]
    if kind == "some of two":
        rows = [sorted({*r, int(rng.integers(0, k))}) if i % 7 == 0 else r for i, r in enumerate(rows)]
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    col = np.concatenate([np.array(r) for r in rows]).astype(np.int32)
    val = rng.uniform(-1, 1, len(col)).astype(np.float32).astype(np.float64)
    return HostCSR(len(rows), k, rp, col, val)


@pytest.mark.parametrize("precision", ["fp64", "fp32w", "fp32c"])
@pytest.mark.parametrize("b", ["sorted", "crowded", "any order"])
@pytest.mark.parametrize("a", ["one", "empty rows too", "some of two"])
def test_rows_of_b(cuda, a, b, precision):
    rng = np.random.default_rng(7)
    B = b_rows(rng, b)
    A = a_rows(rng, B.nrows, a, np.flatnonzero(np.diff(B.rowptr) == 0))
    f = lambda h: HostCSR(h.nrows, h.ncols, h.rowptr, h.col, h.val.astype(np.float32))  # noqa: E731
    dA, dB = (f(A), f(B)) if precision != "fp64" else (A, B)
    dA, dB = dA.to_device(), dB.to_device()
    rp, col, val = oracle.spgemm(A, B)
    bound = oracle.absbound(A, B, rp, col)
    one = nb.spgemm(dA, dB, precision=precision).to_host()
    rp2, nnz = nb.spgemm_symbolic(dA, dB)
    two = nb.spgemm_numeric(dA, dB, rp2, nnz, precision=precision).to_host()
    for c in (one, two):
        assert_same_structure(c.rowptr, c.col, rp, col)
        if precision == "fp32c":  # comp_tol of the stricter entry point
            assert np.all(np.abs(c.val - val) <= 1e-12 * bound)
        else:
            assert_bitwise(c.val, val)


def test_several_products(cuda):
    rng = np.random.default_rng(8)
    pairs = []
    for kind in ("sorted", "crowded", "any order"):
        B = b_rows(rng, kind)
        pairs.append((a_rows(rng, B.nrows, "one", None), B))
    Cs = nb.spgemm_batched([x.to_device() for x, _ in pairs], [y.to_device() for _, y in pairs])
    for (A, B), C in zip(pairs, Cs):
        rp, col, val = oracle.spgemm(A, B)
        C = C.to_host()
        assert_same_structure(C.rowptr, C.col, rp, col)
        assert_bitwise(C.val, val)
