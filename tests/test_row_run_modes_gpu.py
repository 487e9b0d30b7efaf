"""The compensated mode in row runs and bunches: which rows sum in fp32 pairs, the
bound reported for them and the rows in fp64 are the same with and without runs,
for B rows with repeated columns and for rows past the row-group kernels."""
import numpy as np
import pytest

import nsp_b200 as nb
import oracle
from nsp_b200.csr import HostCSR

from conftest import assert_bitwise, assert_same_structure
from test_row_run_cpu import csr
from test_row_run_gpu import NO_RUNS, as32, rounded

pytestmark = pytest.mark.gpu

RUNS = 8  # opts.row_kernel: runs for small products too


def shifted(n, offsets, ncols, rng):
    """Row i holds column i + d for every offset d, in the order given."""
    return rounded(csr([[i + d for d in offsets] for i in range(n)], ncols, rng))


def repeated(rng):
    """B rows of three columns, each listed many times: an entry sums 40 products for each A entry."""
    n = 2600
    return shifted(n, (0, 1, 5), n + 8, rng), shifted(n + 8, (0, 3, 1) * 40, n + 16, rng)


def band(k):
    """Rows of 5 * k entries of C, as many products."""
    def make(rng):
        n = 2200
        return (shifted(n, tuple(range(0, 5 * 128, 128)), n + 600, rng),
                shifted(n + 600, tuple(range(k)), n + 800, rng))
    return make


@pytest.mark.parametrize("make", [repeated, band(102), band(103), band(128)])
def test_pair_rows_are_the_same_without_runs(cuda, make):
    A, B = make(np.random.default_rng(11))
    dA, dB = as32(A).to_device(), as32(B).to_device()
    got, st = nb.spgemm(dA, dB, precision="fp32c", row_kernel=RUNS, return_stats=True)
    _, off = nb.spgemm(dA, dB, precision="fp32c", row_kernel=NO_RUNS, return_stats=True)
    for k in ("rows_redone", "max_row_err", "num_bins"):
        assert st[k] == off[k], k
    rp, col, val = oracle.spgemm(A, B)
    got = got.to_host()
    assert_same_structure(got.rowptr, got.col, rp, col)
    bound = oracle.absbound(A, B, rp, col)
    assert np.all(np.abs(got.val - val) <= (st["max_row_err"] + 2.0**-53 * 600) * bound)
    if st["rows_redone"] == A.nrows:  # exact products, summed in A-row order
        assert_bitwise(got.val, val)
    assert (st["rows_redone"] == 0) == (make is not repeated and np.diff(rp).max() <= 512)
