"""Many rows of few products: below 65,536 rows flat lists count and compute them, from
there on row groups of 8 lanes do (rows of at most 48 products, of at most 16 entries)."""
import numpy as np
import pytest

import nsp_b200 as nb
import oracle
from nsp_b200.csr import HostCSR

from conftest import assert_bitwise, assert_same_structure

pytestmark = pytest.mark.gpu


def rows(lens, ncols, rng):
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    top = int(lens.max())
    col = (rng.integers(0, ncols // top, (len(lens), top)) + np.arange(top) * (ncols // top))
    keep = np.arange(top)[None] < lens[:, None]
    return HostCSR(len(lens), ncols, rp, col[keep].astype(np.int32), rng.uniform(-1, 1, rp[-1]))


@pytest.mark.parametrize("n", [65_535, 65_536, 70_001])
@pytest.mark.parametrize("a,b", [(3, 3), (5, 6), (8, 7)])
def test_products(cuda, n, a, b):
    rng = np.random.default_rng(n + a)
    k = 30_011
    A, B = rows(rng.integers(0, a + 1, n), k, rng), rows(rng.integers(0, b + 1, k), 400, rng)
    dA, dB = A.to_device(), B.to_device()
    rp, col, val = oracle.spgemm(A, B)
    rp2, nnz = nb.spgemm_symbolic(dA, dB)
    for C in (nb.spgemm(dA, dB), nb.spgemm_numeric(dA, dB, rp2, nnz)):
        C = C.to_host()
        assert_same_structure(C.rowptr, C.col, rp, col)
        assert_bitwise(C.val, val)
