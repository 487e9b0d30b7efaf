"""Sums of flat product lists, rows of 513 to 4096 entries (one block a row): in A-row
order from zero, bit for bit the sequential sum, where the list holds the row's
products; the compensated mode within the bound of each entry point."""
import numpy as np
import pytest

import nsp_b200 as nb
import oracle
from nsp_b200.csr import HostCSR

from conftest import assert_bitwise, assert_same_structure

pytestmark = pytest.mark.gpu

# d * d products a row over m columns, 1.12 times as many as entries: bins 6, 7 and 8
SIZES = {6: (28, 3500), 7: (40, 7000), 8: (56, 14000)}


def rows(n, ncols, deg, rng):
    col = np.concatenate([np.sort(rng.choice(ncols, deg, replace=False)) for _ in range(n)])
    val = rng.uniform(-1, 1, n * deg).astype(np.float32).astype(np.float64)
    return HostCSR(n, ncols, np.arange(0, n * deg + 1, deg, dtype=np.int32), col.astype(np.int32), val)


def as32(h):
    return HostCSR(h.nrows, h.ncols, h.rowptr, h.col, h.val.astype(np.float32))


@pytest.mark.parametrize("precision", ["fp64", "fp32w", "fp32c"])
@pytest.mark.parametrize("bin_", SIZES)
def test_sums_in_order(cuda, bin_, precision):
    rng = np.random.default_rng(bin_)
    d, m = SIZES[bin_]
    A, B = rows(300, 500, d, rng), rows(500, m, d, rng)
    dA, dB = (A, B) if precision == "fp64" else (as32(A), as32(B))
    dA, dB = dA.to_device(), dB.to_device()
    rp, col, val = oracle.spgemm(A, B)
    one, st = nb.spgemm(dA, dB, precision=precision, return_stats=True)
    assert st["num_bins"][bin_] == A.nrows and st["intprod"] < 1.25 * st["nnz"]
    rp2, nnz = nb.spgemm_symbolic(dA, dB)
    two = nb.spgemm_numeric(dA, dB, rp2, nnz, precision=precision)
    bound = oracle.absbound(A, B, rp, col)
    for C, tol in ((one, 1e-10), (two, 1e-12)):  # comp_tol of the two entry points
        C = C.to_host()
        assert_same_structure(C.rowptr, C.col, rp, col)
        if precision == "fp32c":
            assert np.all(np.abs(C.val - val) <= tol * bound)
        else:
            assert_bitwise(C.val, val)
