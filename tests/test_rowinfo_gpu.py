"""Products of every row (k_rowinfo, k_rowinfo_group, k_rowinfo_long) against numpy: at
the row counts and row lengths where the kernels change, B the same matrix or another
(its order is checked on the way), and several products with tiles across their rows."""
import numpy as np
import pytest

import nsp_b200 as nb
import oracle
from nsp_b200.csr import HostCSR

from conftest import assert_bitwise, assert_same_structure

pytestmark = pytest.mark.gpu


def csr(lens, ncols, rng):
    """Rows of these lengths, columns ascending from a random start, wrapped into order."""
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    step = max(ncols // (int(max(lens)) + 1), 1)
    col = [np.sort((int(rng.integers(0, ncols)) + step * np.arange(d)) % ncols) for d in lens]
    col = np.concatenate(col).astype(np.int32)
    return HostCSR(len(lens), ncols, rp, col, rng.uniform(-1, 1, rp[-1]))


LENGTHS = {
    "short": lambda rng, n: rng.integers(0, 13, n),
    "to a warp": lambda rng, n: rng.choice([0, 1, 63, 64, 65, 66], n),
    "to a block": lambda rng, n: np.where(rng.random(n) < 0.002, rng.choice([1023, 1024, 1025, 3000], n),
                                          rng.integers(0, 9, n)),
    "long": lambda rng, n: rng.integers(60, 90, n),
}


@pytest.mark.parametrize("kind", LENGTHS)
@pytest.mark.parametrize("n", [1, 255, 15999, 16000, 16257])
def test_row_products(cuda, n, kind):
    rng = np.random.default_rng(n)
    k = 6007
    A = csr(LENGTHS[kind](rng, n), k, rng)
    B = csr(rng.integers(0, 20, k), 900, rng)
    rows, total = nb.intprod(A.to_device(), B.to_device())
    blen = np.diff(B.rowptr).astype(np.int64)
    want = np.concatenate([[0], np.cumsum(blen[A.col])])
    want = want[A.rowptr[1:]] - want[A.rowptr[:-1]]
    assert np.array_equal(np.asarray(rows.cpu()), want)
    assert total == want.sum()


@pytest.mark.parametrize("n", [2000, 17000])
def test_order_is_checked_on_the_way(cuda, n):
    rng = np.random.default_rng(3)
    lens = rng.choice([0, 2, 63, 64, 65, 100], n, p=[.2, .5, .1, .05, .05, .1])
    A = csr(lens, n, rng)
    rows = [r for r in range(n) if lens[r] >= 2]
    d = A.to_device()
    _, st = nb.spgemm(d, d, return_stats=True)
    assert st["b_sorted"] == 1
    for r in (rows[0], rows[-1], int(np.argmax(lens)), int(np.nonzero(lens == 64)[0][0])):
        col = A.col.copy()
        e = int(A.rowptr[r + 1])
        col[e - 2], col[e - 1] = col[e - 1], col[e - 2]
        d = HostCSR(n, n, A.rowptr, col, A.val).to_device()
        _, st = nb.spgemm(d, d, return_stats=True)
        assert st["b_sorted"] == 0, r


def test_tiles_across_products(cuda):
    rng = np.random.default_rng(4)
    pairs = []
    for n in (4097, 5001, 33, 7500):
        k = 700
        A = csr(rng.choice([0, 1, 5, 64, 65, 130], n, p=[.2, .4, .3, .04, .03, .03]), k, rng)
        pairs.append((A, csr(rng.integers(0, 6, k), 5000, rng)))
    Cs = nb.spgemm_batched([a.to_device() for a, _ in pairs], [b.to_device() for _, b in pairs])
    for (A, B), C in zip(pairs, Cs):
        rp, col, val = oracle.spgemm(A, B)
        C = C.to_host()
        assert_same_structure(C.rowptr, C.col, rp, col)
        keep = np.repeat(np.diff(rp) <= 512, np.diff(rp))
        assert_bitwise(C.val[keep], val[keep])
