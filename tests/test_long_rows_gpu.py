"""Rows of C that a block works on (k_num_block, k_num_rank, k_sym_wide) over B rows
whose mean length lies on either side of the lines between the two walks of a row's
products: B rows of one length at the lines, and mixes of empty, short, medium and
block-long rows. Two-call steps take B's own mean row."""
import numpy as np
import pytest

import nsp_b200 as nb
import oracle
from nsp_b200.csr import HostCSR

from conftest import assert_same_structure

pytestmark = pytest.mark.gpu


def rows(lens, ncols, rng, fp32):
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    col = np.concatenate([np.sort(rng.choice(ncols, d, replace=False)) for d in lens])
    val = rng.uniform(-1, 1, rp[-1])
    return HostCSR(len(lens), ncols, rp, col.astype(np.int32),
                   val.astype(np.float32).astype(np.float64) if fp32 else val)


def as32(h):
    return HostCSR(h.nrows, h.ncols, h.rowptr, h.col, h.val.astype(np.float32))


def mixed(rng, k):
    return rng.choice([0, 1, 4, 5, 16, 17, 31, 33, 64, 200, 1023, 1024, 1025, 2500], k,
                      p=[.05, .1, .1, .1, .1, .1, .1, .1, .1, .1, .02, .01, .01, .01])


B_ROWS = {"56": 56, "57": 57, "128": 128, "129": 129, "300": 300, "mixed": mixed}


@pytest.mark.parametrize("b", B_ROWS)
@pytest.mark.parametrize("ncols", [900, 3500, 60_000])  # rows of <= 1024, <= 4096, more entries
@pytest.mark.parametrize("precision", ["fp64", "fp32w"])
def test_both_walks(cuda, b, ncols, precision):
    rng = np.random.default_rng(len(b) + ncols)
    k, fp32 = 1100, precision != "fp64"
    lens = B_ROWS[b](rng, k) if callable(B_ROWS[b]) else np.full(k, B_ROWS[b])
    B = rows(np.minimum(lens, ncols), ncols, rng, fp32)
    # rounds of a few entries, of 255..257, 1023..1025, and two rounds and a rest
    A = rows([0, 1, 15, 16, 40, 63, 64, 65, 255, 256, 257, 511, 513, 1023, 1024, 1025, 1100] * 2,
             k, rng, fp32)
    A.col[A.rowptr[-2]:] = np.sort(rng.integers(0, k, 1100))  # columns repeated in A
    dA, dB = (as32(A), as32(B)) if fp32 else (A, B)
    dA, dB = dA.to_device(), dB.to_device()
    rp, col, val = oracle.spgemm(A, B)
    bound = oracle.absbound(A, B, rp, col)
    terms = 1100  # at most: one product of an entry for each A entry
    one = nb.spgemm(dA, dB, precision=precision).to_host()
    rp2, nnz = nb.spgemm_symbolic(dA, dB)
    two = nb.spgemm_numeric(dA, dB, rp2, nnz, precision=precision).to_host()
    for c in (one, two):
        assert_same_structure(c.rowptr, c.col, rp, col)
        assert np.all(np.abs(c.val - val) <= 2 * terms * 2.0**-53 * bound)


def test_batch(cuda):
    rng = np.random.default_rng(9)
    pairs = []
    for k, m, d in ((300, 50_000, 200), (200, 2000, 300), (400, 9000, 70)):
        pairs.append((rows(rng.integers(0, 200, 60), k, rng, False),
                      rows(np.full(k, d), m, rng, False)))
    Cs = nb.spgemm_batched([a.to_device() for a, _ in pairs], [b.to_device() for _, b in pairs])
    for (A, B), C in zip(pairs, Cs):
        rp, col, val = oracle.spgemm(A, B)
        C = C.to_host()
        assert_same_structure(C.rowptr, C.col, rp, col)
        assert np.all(np.abs(C.val - val) <= 2 * 200 * 2.0**-53 * oracle.absbound(A, B, rp, col))
