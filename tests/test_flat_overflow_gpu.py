"""Rows with more products than their flat list holds, all rows of a product or some of
them, in every bin that has lists: they are computed by the hash kernel of their bin."""
import numpy as np
import pytest

import nsp_b200 as nb
import oracle
from nsp_b200.csr import HostCSR

from conftest import assert_bitwise, assert_same_structure

pytestmark = pytest.mark.gpu


def rows(n, ncols, deg, rng, first=0):
    col = np.concatenate([first + np.sort(rng.choice(ncols, deg, replace=False)) for _ in range(n)])
    return col.astype(np.int32), rng.uniform(-1, 1, n * deg).astype(np.float32).astype(np.float64)


def product(parts, rng, n=250, k=400):
    """A rows of d entries over B rows of d entries within m columns, for each (d, m)."""
    ac, av, bc, bv, al, bl = [], [], [], [], [], []
    cols = 0
    for i, (d, m) in enumerate(parts):
        c, v = rows(n, k, d, rng, i * k)
        ac.append(c); av.append(v); al += [d] * n
        c, v = rows(k, m, d, rng, cols)
        bc.append(c); bv.append(v); bl += [d] * k
        cols += m

    def csr(lens, ncols, c, v):
        rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
        return HostCSR(len(lens), ncols, rp, np.concatenate(c), np.concatenate(v))
    return csr(al, k * len(parts), ac, av), csr(bl, cols, bc, bv)


# (d, m): d * d products a row, just more than the bin's list holds, with about 0.72 times as
# many entries, in the upper part of the bin
OVER = {3: (13, 230), 4: (18, 473), 5: (26, 926), 6: (37, 1928), 7: (52, 3947), 8: (72, 8569)}


def as32(h):
    return HostCSR(h.nrows, h.ncols, h.rowptr, h.col, h.val.astype(np.float32))


def check(A, B, precision):
    dA, dB = (A, B) if precision == "fp64" else (as32(A), as32(B))
    dA, dB = dA.to_device(), dB.to_device()
    rp, col, val = oracle.spgemm(A, B)
    bound = oracle.absbound(A, B, rp, col)
    one, st = nb.spgemm(dA, dB, precision=precision, return_stats=True)
    rp2, nnz = nb.spgemm_symbolic(dA, dB)
    two = nb.spgemm_numeric(dA, dB, rp2, nnz, precision=precision)
    tol = 1e-10 if precision == "fp32c" else 2.0**-53 * 2 * 100  # 72 terms at most
    for C in (one, two):
        C = C.to_host()
        assert_same_structure(C.rowptr, C.col, rp, col)
        assert np.all(np.abs(C.val - val) <= tol * bound)
        if precision != "fp32c":
            keep = np.repeat(np.diff(rp) <= 512, np.diff(rp))
            assert_bitwise(C.val[keep], val[keep])
    if precision == "fp32c":  # rows of the row-group bins in pairs, the others in fp64
        assert st["rows_redone"] == int(np.sum(np.diff(rp) > 512))
    return st


@pytest.mark.parametrize("precision", ["fp64", "fp32w", "fp32c"])
@pytest.mark.parametrize("bin_", OVER)
def test_every_row(cuda, bin_, precision):
    rng = np.random.default_rng(bin_)
    A, B = product([OVER[bin_]], rng)
    st = check(A, B, precision)
    assert st["num_bins"][bin_] > 0.9 * A.nrows  # the bin this is about
    assert 1.25 < st["intprod"] / st["nnz"] < 1.5


def test_some_rows_of_every_bin(cuda):
    rng = np.random.default_rng(40)
    parts = [OVER[b] for b in OVER] + [(d, 40 * m) for d, m in OVER.values()]
    check(*product(parts, rng, n=40, k=90), "fp64")
    # few of them among many rows that fit: one kernel for the bins of a kind
    parts = [(d, 60 * m) for d, m in OVER.values()] * 3 + [OVER[3], OVER[4]]
    A, B = product(parts, rng, n=60, k=90)
    st = check(A, B, "fp64")
    assert st["intprod"] <= 1.05 * st["nnz"]
