"""Rows whose products are one flat list: counted (k_sym_flat, row_products) and,
where few columns repeat, sorted (k_num_flat). Sums are formed in A-row order from zero, like the oracle's,
so values are compared bit for bit. Sizes: row lengths at the edges of the
bins and of the lists, empty rows of A and B, B rows longer than a block,
repeated columns inside a bucket and at the ends of a row, rows whose columns
crowd a few buckets, rows with more
products than a list holds (left to the hash kernels), B rows in any order."""
import numpy as np
import pytest

import nsp_b200 as nb
import oracle
from nsp_b200.csr import HostCSR

from conftest import assert_bitwise, assert_same_structure

pytestmark = pytest.mark.gpu


def from_rows(rows, ncols, rng, shuffled=False):
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    col = np.concatenate([r if shuffled else np.sort(r) for r in rows]) if rp[-1] else np.zeros(0)
    val = rng.uniform(-1, 1, rp[-1]).astype(np.float32).astype(np.float64)
    return HostCSR(len(rows), ncols, rp, col.astype(np.int32), val)


def pick(rng, n, k):
    return rng.choice(n, size=k, replace=False)


def edges(rng):
    """B rows of one entry, all columns different: products and entries of a row are A's degree."""
    k = 9000
    lens = [0, 1, 2, 3]
    for e in (16, 32, 64, 128, 160, 256, 320, 512, 640, 1024, 1280, 2048, 2560, 4096):
        lens += [e - 1, e, e + 1]
    lens += [5119, 5120, 5121, 8000]
    A = from_rows([pick(rng, k, d) for d in lens], k, rng)
    m = 50_021
    B = from_rows([c[None] for c in pick(rng, m, k)], m, rng)
    return A, B


def mixed(rng, shuffled=False):
    """Random rows, empty ones, hubs of B, and a few rows of A whose products nearly all meet."""
    n, k, m = 700, 900, 30_011
    brows = [pick(rng, m, rng.integers(0, 40)) for _ in range(k - 40)]
    brows += [pick(rng, m, 700 + 60 * i) for i in range(4)]
    brows += [pick(rng, 60, 30) for _ in range(36)]  # columns 0..59 only
    arows = [pick(rng, k - 40, rng.integers(0, 60)) for _ in range(n)]
    for i in range(4):
        arows[7 * i] = np.append(pick(rng, k - 40, 3 + i), k - 40 + i)      # a hub of B
    for i in range(9):
        arows[11 * i + 3] = np.arange(k - 36, k)[: 4 * (i + 1)]               # 60 columns at most
    arows[500] = np.concatenate([pick(rng, k - 40, 200), np.arange(k - 40, k)])
    return from_rows(arows, k, rng), from_rows(brows, m, rng, shuffled)


def clusters(rng):
    """Columns side by side, far from the others of the row: crowded buckets."""
    k, m = 800, 400_009
    start = rng.integers(0, m - 40, k)
    B = from_rows([s + np.arange(rng.integers(1, 40)) for s in start], m, rng)
    A = from_rows([pick(rng, k, rng.integers(1, 200)) for _ in range(300)], k, rng)
    return A, B


def counts(rng):
    """Products at the edges of the symbolic bins; rows with many more products than C has columns."""
    lens = [d for e in (24, 48, 96, 192, 384, 768, 1536, 3072, 6144) for d in (e - 1, e, e + 1)]
    k, m = 7000, 40_009
    A = from_rows([pick(rng, k, d) for d in lens], k, rng)
    B = from_rows([c[None] for c in pick(rng, m, k)], m, rng)
    return A, B


def narrow(rng):
    k, m = 500, 33
    B = from_rows([pick(rng, m, rng.integers(0, 20)) for _ in range(k)], m, rng)
    A = from_rows([pick(rng, k, d) for d in (0, 1, 2, 3, 4, 40, 100, 300, 500)], k, rng)
    return A, B


def heavy(rng):
    """Rounds of over 16384 products, of 1024 entries and of one more, B rows of 1024 entries."""
    k, m = 3000, 300_007
    brows = [pick(rng, m, rng.integers(0, 60)) for _ in range(k - 4)]
    brows += [pick(rng, m, d) for d in (1023, 1024, 1025, 5000)]
    arows = [pick(rng, k - 4, d) for d in (300, 1023, 1024, 1025, 2500)]
    arows += [np.append(pick(rng, k - 4, d), np.arange(k - 4, k)) for d in (0, 200, 1020, 1024)]
    return from_rows(arows, k, rng), from_rows(brows, m, rng)


def as32(h):
    return HostCSR(h.nrows, h.ncols, h.rowptr, h.col, h.val.astype(np.float32))


def check(A, B, precision, exact=True):
    X, Y = (A, B) if precision == "fp64" else (as32(A), as32(B))
    dA, dB = X.to_device(), Y.to_device()
    C = nb.spgemm(dA, dB, precision=precision).to_host()
    rp2, nnz = nb.spgemm_symbolic(dA, dB)
    C2 = nb.spgemm_numeric(dA, dB, rp2, nnz, precision=precision).to_host()
    rp, col, val = oracle.spgemm(A, B)
    bound = oracle.absbound(A, B, rp, col)
    tol = {"fp64": 2.0**-50, "fp32w": 2.0**-50, "fp32c": 1e-10}[precision]
    for c in (C, C2):
        assert_same_structure(c.rowptr, c.col, rp, col)
        assert np.all(np.abs(c.val - val) <= tol * np.maximum(bound, 1e-300) * 40)
        # longer rows of many products of few columns take kernels that add in any order
        if exact and precision != "fp32c":
            keep = np.repeat(np.diff(rp) <= 512, np.diff(rp))
            assert_bitwise(c.val[keep], val[keep])


@pytest.mark.parametrize("precision", ["fp64", "fp32w", "fp32c"])
@pytest.mark.parametrize("make", [edges, mixed, clusters, counts, narrow, heavy])
def test_rows(cuda, make, precision):
    check(*make(np.random.default_rng(5)), precision)


def test_b_in_any_order(cuda):
    check(*mixed(np.random.default_rng(6), shuffled=True), "fp64", exact=False)


def test_batch(cuda):
    pairs = [mixed(np.random.default_rng(20 + i)) for i in range(3)]
    pairs.append(edges(np.random.default_rng(30)))
    Cs = nb.spgemm_batched([a.to_device() for a, _ in pairs], [b.to_device() for _, b in pairs])
    for (A, B), C in zip(pairs, Cs):
        rp, col, val = oracle.spgemm(A, B)
        C = C.to_host()
        assert_same_structure(C.rowptr, C.col, rp, col)
        keep = np.repeat(np.diff(rp) <= 512, np.diff(rp))
        assert_bitwise(C.val[keep], val[keep])
