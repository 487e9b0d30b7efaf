"""Whose memory a kept output block is: blocks of the same address and size that
belong to someone else, and threads that have made no CUDA call yet."""
import ctypes as C
import threading

import pytest

import nsp_b200 as nb
from nsp_b200._lib import lib

from test_out_pool_gpu import product, ptrs, rt

pytestmark = pytest.mark.gpu


def test_same_address_and_size_of_someone_else(cuda):
    """Kept blocks that their caller frees as well; another allocator is given their
    addresses with their sizes and keeps its data through the next product."""
    import torch
    assert lib.nspb_trim() == 0
    A = nb.gen.stencil(40, npts=27).to_device()
    c = product(A)
    nbytes = [4 * (A.nrows + 1), 4 * c.nnz, 8 * c.nnz]
    sizes = [(n + 511) // 512 * 512 for n in nbytes]
    for p in ptrs(c):
        assert lib.nspb_free(p) == 0
    for p in ptrs(c):
        assert rt.cudaFree(C.c_void_p(p)) == 0
    held = []
    for n in sizes:
        q = C.c_void_p()
        assert rt.cudaMalloc(C.byref(q), C.c_size_t(n)) == 0
        assert rt.cudaMemset(q, 0x5a, C.c_size_t(n)) == 0
        held.append(q.value)
    assert set(held) & set(ptrs(c))  # the case this is about: an address came back
    d = product(A)
    assert not set(held) & set(ptrs(d))
    torch.cuda.synchronize()
    for q, n in zip(held, sizes):
        host = (C.c_ubyte * n)()
        assert rt.cudaMemcpy(host, C.c_void_p(q), C.c_size_t(n), 2) == 0
        assert bytes(host) == b"\x5a" * n
    for p in ptrs(d) + held:
        assert lib.nspb_free(p) == 0
    assert lib.nspb_trim() == 0


def test_trim_in_a_new_thread_gives_the_memory_back(cuda):
    import torch
    A = nb.gen.stencil(64, npts=27).to_device()
    assert lib.nspb_trim() == 0
    c = product(A)
    for p in ptrs(c):
        assert lib.nspb_free(p) == 0
    torch.cuda.synchronize()
    kept = torch.cuda.mem_get_info()[0]
    r = []
    t = threading.Thread(target=lambda: r.append(lib.nspb_trim()))
    t.start()
    t.join()
    assert r == [0]
    assert torch.cuda.mem_get_info()[0] - kept >= 32 << 20


@pytest.mark.parametrize("mode", [1, 2])  # another thread's thread-local capture, a relaxed one
def test_captures_go_on(cuda, mode):
    """An output is freed while another thread captures a stream: the capture is whole."""
    A = nb.gen.stencil(20, npts=27).to_device()
    c = product(A)
    s, g = C.c_void_p(), C.c_void_p()
    assert rt.cudaStreamCreateWithFlags(C.byref(s), 1) == 0
    assert rt.cudaStreamBeginCapture(s, mode) == 0
    r = []
    t = threading.Thread(target=lambda: r.extend(lib.nspb_free(p) for p in ptrs(c)))
    t.start()
    t.join()
    end = rt.cudaStreamEndCapture(s, C.byref(g))
    rt.cudaGetLastError()
    assert r == [0, 0, 0] and end == 0
    assert rt.cudaGraphDestroy(g) == 0 and rt.cudaStreamDestroy(s) == 0


def test_plans_are_made_while_outputs_are_freed(cuda):
    A = nb.gen.stencil(12, npts=27).to_device()
    stop, made = threading.Event(), []

    def products():
        while not stop.is_set():
            for p in ptrs(product(A)):
                made.append(lib.nspb_free(p))
    t = threading.Thread(target=products)
    t.start()
    try:
        for _ in range(60):
            nb.Plan([A], [A]).execute()
    finally:
        stop.set()
        t.join()
    assert made and not any(made)
