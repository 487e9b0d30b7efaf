"""Long rows of A over B rows of a few entries: rounds of A entries that make no list of
products (every B row of at most 2 entries, or 6 in launches of at most 16 rows), beside
rounds that make one, in k_sym_wide and k_num_rank (rows of more than 4096 entries) and
k_num_block."""
import numpy as np
import pytest

import nsp_b200 as nb
import oracle
from nsp_b200.csr import HostCSR

from conftest import assert_same_structure

pytestmark = pytest.mark.gpu

K, M = 24_000, 30_011


def rows(lens, ncols, rng, order=None):
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    cols = [np.sort(rng.choice(ncols, d, replace=False)) for d in lens]
    val = rng.uniform(-1, 1, rp[-1]).astype(np.float32).astype(np.float64)
    return HostCSR(len(lens), ncols, rp, np.concatenate(cols).astype(np.int32), val)


def blocks(rng, n):
    """B rows of one length for a stretch, so that a round of A's entries has one kind or two."""
    out, kinds = np.zeros(n, int), [0, 1, 2, 3, 6, 7, 30, 1100]
    i = 0
    while i < n:
        w = int(rng.integers(200, 4000))
        out[i:i + w] = rng.choice(kinds, p=[.15, .15, .2, .15, .15, .1, .09, .01])
        i += w
    return out


@pytest.mark.parametrize("count", [1, 16, 17])
@pytest.mark.parametrize("b", [1, 2, 3, 6, 7, "blocks"])
@pytest.mark.parametrize("precision", ["fp64", "fp32w"])
def test_rounds_without_a_list(cuda, count, b, precision):
    rng = np.random.default_rng(count)
    lens = blocks(rng, K) if b == "blocks" else np.full(K, b)
    B = rows(lens, M, rng)
    degrees = [12_000, 8193, 9000, 10_240, 7169, 20_000]
    A = rows([degrees[i % 6] for i in range(count)], K, rng)
    f = lambda h: HostCSR(h.nrows, h.ncols, h.rowptr, h.col, h.val.astype(np.float32))  # noqa: E731
    dA, dB = (f(A), f(B)) if precision == "fp32w" else (A, B)
    dA, dB = dA.to_device(), dB.to_device()
    rp, col, val = oracle.spgemm(A, B)
    bound = oracle.absbound(A, B, rp, col)
    one = nb.spgemm(dA, dB, precision=precision).to_host()
    rp2, nnz = nb.spgemm_symbolic(dA, dB)
    two = nb.spgemm_numeric(dA, dB, rp2, nnz, precision=precision).to_host()
    for c in (one, two):
        assert_same_structure(c.rowptr, c.col, rp, col)
        assert np.all(np.abs(c.val - val) <= 2 * 20_000 * 2.0**-53 * bound)  # a term an A entry


def test_rows_of_a_block(cuda):
    """k_num_block: rows of 513 to 4096 entries with many products each."""
    rng = np.random.default_rng(3)
    for d in (1, 2, 3):
        A, B = rows([1500, 2900, 1025, 0, 2048] * 8, 3000, rng), rows(np.full(3000, d), 900, rng)
        C = nb.spgemm(A.to_device(), B.to_device()).to_host()
        rp, col, val = oracle.spgemm(A, B)
        assert_same_structure(C.rowptr, C.col, rp, col)
        assert np.all(np.abs(C.val - val) <= 2 * 2900 * 2.0**-53 * oracle.absbound(A, B, rp, col))
