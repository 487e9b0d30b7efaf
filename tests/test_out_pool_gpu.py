"""Blocks of outputs that the library allocates are kept by nspb_free for later
outputs: reuse, what is not reused (a block freed with cudaFree, or twice), the
order of a block's last reader and its next owner, and giving all back."""
import ctypes as C

import numpy as np
import pytest

import nsp_b200 as nb
import oracle
from nsp_b200._lib import CsrOut, lib

from conftest import assert_bitwise, assert_same_structure

pytestmark = pytest.mark.gpu

rt = C.CDLL("libcudart.so.12")


def product(A):
    a, c, o = A.as_in(), CsrOut(), nb.make_opts()
    assert lib.nspb_spgemm(C.byref(a), C.byref(a), C.byref(c), C.byref(o), None) == 0
    return c


def ptrs(c):
    return [c.rowptr, c.col, c.val]


@pytest.mark.parametrize("L", [9, 40])  # blocks inside one driver chunk, and of their own
def test_blocks_come_back(cuda, L):
    assert lib.nspb_trim() == 0
    H = nb.gen.stencil(L, npts=27)
    A = H.to_device()
    first = product(A)
    for p in ptrs(first):
        assert lib.nspb_free(p) == 0
        assert lib.nspb_free(p) != 0  # kept: not free a second time
    second = product(A)
    assert sorted(ptrs(second)) == sorted(ptrs(first))
    rp, col, val = oracle.spgemm(H, H)
    got = nb.DeviceCSR(second.nrows, second.ncols, nb.adopt(second.rowptr, second.nrows + 1, "int32"),
                       nb.adopt(second.col, second.nnz, "int32"),
                       nb.adopt(second.val, second.nnz, "float64")).to_host()
    assert_same_structure(got.rowptr, got.col, rp, col)
    assert_bitwise(got.val, val)


def test_cuda_free_works_and_is_noticed(cuda):
    assert lib.nspb_trim() == 0
    A = nb.gen.stencil(24, npts=27).to_device()
    c = product(A)
    for p in ptrs(c):
        assert rt.cudaFree(C.c_void_p(p)) == 0
    # the addresses belong to someone else now: freeing them leaves their data alone
    held = [C.c_void_p() for _ in range(3)]
    for h in held:
        assert rt.cudaMalloc(C.byref(h), C.c_size_t(96 << 20)) == 0
    d = product(A)
    for p in ptrs(d):
        assert lib.nspb_free(p) == 0
    for p in ptrs(d):  # a block that is kept, freed by its caller all the same
        assert rt.cudaFree(C.c_void_p(p)) == 0
    e = product(A)
    assert lib.nspb_trim() == 0
    for p in ptrs(e) + [h.value for h in held]:
        assert lib.nspb_free(p) == 0
    assert lib.nspb_trim() == 0


def test_free_waits_for_readers(cuda):
    import torch
    A = nb.gen.stencil(60, npts=27).to_device()
    s = torch.cuda.Stream()
    want = None
    for _ in range(3):
        Cm = nb.spgemm(A, A)
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s):  # long reads of C on another stream, then C goes
            tot = torch.zeros((), dtype=torch.float64, device="cuda")
            for _ in range(20):
                tot = tot + Cm.val.abs().sum()
        del Cm
        nb.spgemm(A, nb.DeviceCSR(A.nrows, A.ncols, A.rowptr, A.col, A.val * 3.0))
        s.synchronize()
        want = want if want is not None else float(tot)
        assert float(tot) == want


def test_trim_gives_the_memory_back(cuda):
    import torch
    A = nb.gen.stencil(64, npts=27).to_device()
    assert lib.nspb_trim() == 0
    torch.cuda.synchronize()
    product_free = torch.cuda.mem_get_info()[0]
    C1 = nb.spgemm(A, A)
    del C1
    kept_free = torch.cuda.mem_get_info()[0]
    assert lib.nspb_trim() == 0
    assert torch.cuda.mem_get_info()[0] - kept_free >= 32 << 20
    assert kept_free < product_free
