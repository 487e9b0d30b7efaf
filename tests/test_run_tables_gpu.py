"""More patterns than the tables of the row runs hold: of runs (each block of rows has its
own), of the rows left over (half of a grid's rows at random, in one stretch or
scattered), in one product, a batch and a plan. What finds no place is computed by the
other kernels; values are sums in A-row order either way."""
import numpy as np
import pytest

import nsp_b200 as nb
import oracle
from nsp_b200.csr import HostCSR

from conftest import assert_bitwise, assert_same_structure

pytestmark = pytest.mark.gpu

RUNS = 8  # opts.row_kernel: runs for small products too


def grid_with_random_rows(rng, dims, random_rows):
    """A 7-point grid, and the same with these rows at random columns, no two alike."""
    B = nb.gen.stencil(*dims, npts=7)
    col = B.col.copy()
    for i in np.nonzero(random_rows)[0]:
        s, e = B.rowptr[i], B.rowptr[i + 1]
        col[s:e] = np.sort(rng.choice(B.ncols, e - s, replace=False))
    return HostCSR(B.nrows, B.ncols, B.rowptr, col, B.val), B


def blocks(rng, count, rows=7, entries=4, n=4000):
    """Blocks of rows that move by one column, every block with its own columns."""
    off = np.sort(rng.integers(0, n - rows, (count, entries)), 1)
    off += np.arange(entries)  # no two alike
    col = (off[:, None, :] + np.arange(rows)[None, :, None]).reshape(-1)
    m = count * rows
    A = HostCSR(m, n + entries + rows, (np.arange(m + 1) * entries).astype(np.int32),
                col.astype(np.int32), rng.uniform(-1, 1, m * entries))
    k = A.ncols
    bc = (np.arange(k)[:, None] + np.array([0, 3, 9])[None]).reshape(-1)
    return A, HostCSR(k, k + 9, (np.arange(k + 1) * 3).astype(np.int32), bc.astype(np.int32),
                      rng.uniform(-1, 1, 3 * k))


def cases(rng):
    dims = (40, 20, 18)
    n = dims[0] * dims[1] * dims[2]
    i = np.arange(n)
    return {"stretch": grid_with_random_rows(rng, dims, i >= 0.6 * n),
            "scattered": grid_with_random_rows(rng, dims, i % 40 >= 25),
            "few": grid_with_random_rows(rng, dims, i % 997 == 5),
            "runs": blocks(rng, 4600),
            "short runs left": blocks(rng, 900, rows=8)}


@pytest.mark.parametrize("case", ["stretch", "scattered", "few", "runs", "short runs left"])
def test_products(cuda, case):
    A, B = cases(np.random.default_rng(3))[case]
    dA, dB = A.to_device(), B.to_device()
    rp, col, val = oracle.spgemm(A, B)
    for _ in range(2):  # which rows find a place differs from run to run
        C = nb.spgemm(dA, dB, row_kernel=RUNS).to_host()
        assert_same_structure(C.rowptr, C.col, rp, col)
        assert_bitwise(C.val, val)


def test_two_calls_batch_and_plan(cuda, monkeypatch):
    monkeypatch.setenv("NSPB_ROW_KERNEL", str(RUNS))
    pairs = list(cases(np.random.default_rng(4)).values())
    dA, dB = [a.to_device() for a, _ in pairs], [b.to_device() for _, b in pairs]
    want = [oracle.spgemm(a, b) for a, b in pairs]

    def check(C, w, scale=1.0):
        C = C.to_host()
        assert_same_structure(C.rowptr, C.col, w[0], w[1])
        assert_bitwise(C.val, scale * w[2])
    for a, b, w in zip(dA, dB, want):
        rp, nnz = nb.spgemm_symbolic(a, b)
        check(nb.spgemm_numeric(a, b, rp, nnz), w)
    for C, w in zip(nb.spgemm_batched(dA, dB), want):
        check(C, w)
    plan = nb.Plan(dA, dB)
    for a in dA:
        a.val.mul_(-2.0)
    plan.execute()
    for C, w in zip(plan.C, want):
        check(C, w, -2.0)
