"""The blocks that nspb_free keeps (outpool.cpp), built against a CUDA runtime
that only hands out addresses: whose memory a block is, and from which thread."""
import ctypes as C
import os
import subprocess
import sys
import threading

import pytest

from conftest import ROOT

MB = 1 << 20


@pytest.fixture(scope="module")
def built(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("pool") / "libpool.so")
    csrc = os.path.join(ROOT, "nsp_b200", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-pthread", "-shared", "-fPIC",
                    "-Wl,-Bsymbolic", "-I", csrc, "-I", "/usr/local/cuda/include",
                    os.path.join(csrc, "outpool.cpp"),
                    os.path.join(ROOT, "tests", "native", "fake_runtime.cpp"), "-o", so], check=True)
    return so


@pytest.fixture
def pool(built):
    lib = C.CDLL(built)
    lib.fake_malloc.restype = C.c_void_p
    lib.fake_malloc.argtypes = lib.fake_capacity.argtypes = [C.c_size_t]
    lib.fake_free.argtypes = lib.nspb_free.argtypes = [C.c_void_p]
    lib.fake_used.restype = C.c_size_t
    for f in (lib.fake_scratch, lib.fake_device, lib.fake_alloc_out):
        f.argtypes = [C.POINTER(C.c_void_p), C.c_size_t]
    lib.fake_capacity(180 << 30)
    assert lib.nspb_trim() == 0 and lib.fake_used() == 0
    yield lib
    lib.fake_capacity(180 << 30)
    assert lib.nspb_trim() == 0 and lib.fake_used() == 0


def out(lib, nbytes):
    p = C.c_void_p()
    return p.value if lib.fake_alloc_out(C.byref(p), nbytes) == 0 else None


def elsewhere(f):
    """f in a thread of its own."""
    r = []
    t = threading.Thread(target=lambda: r.append(f()))
    t.start()
    t.join()
    return r[0]


def test_kept_blocks_are_given_out_again(pool):
    p = out(pool, 40 * MB)
    assert pool.nspb_free(p) == 0
    assert pool.nspb_free(p) != 0
    assert out(pool, 39 * MB) == p
    assert pool.nspb_free(p) == 0


@pytest.mark.parametrize("taken_by", ["alloc", "trim"])
def test_memory_of_someone_else_at_a_kept_address(pool, taken_by):
    """The caller frees a kept block with cudaFree as well; another allocator of the
    process is given the same address and the same size."""
    p = out(pool, 40 * MB)
    assert pool.nspb_free(p) == 0
    assert pool.fake_free(p) == 0
    theirs = pool.fake_malloc(40 * MB)
    assert theirs == p
    if taken_by == "alloc":
        q = out(pool, 40 * MB)
        assert q != theirs
        assert pool.nspb_free(q) == 0
    assert pool.nspb_trim() == 0
    assert pool.fake_used() == 40 * MB  # theirs is still allocated
    assert pool.fake_free(theirs) == 0


def test_freed_by_its_owner_then_someone_elses(pool):
    """An output that went to cudaFree: a later block at its address is not kept."""
    p = out(pool, 40 * MB)
    assert pool.fake_free(p) == 0
    theirs = pool.fake_malloc(40 * MB)
    assert theirs == p
    assert pool.nspb_free(theirs) == 0  # any cudaMalloc block: to cudaFree
    assert pool.fake_used() == 0


@pytest.mark.parametrize("use", ["alloc", "trim", "free"])
def test_a_thread_without_a_context(pool, use):
    """Kept blocks reach a thread that has made no CUDA call yet: none is lost."""
    p = out(pool, 40 * MB)
    if use != "free":
        assert pool.nspb_free(p) == 0

    def other():
        pool.fake_no_context()
        if use == "alloc":
            return out(pool, 40 * MB)
        return pool.nspb_trim() if use == "trim" else pool.nspb_free(p)
    got = elsewhere(other)
    if use == "alloc":
        assert got == p
        assert pool.nspb_free(p) == 0
    else:
        assert got == 0
    if use == "trim":
        assert pool.fake_used() == 0
    else:
        assert out(pool, 40 * MB) == p
        assert pool.nspb_free(p) == 0


def test_a_capture_elsewhere_goes_on(pool):
    """nspb_free during another thread's thread-local capture, or a relaxed one: allowed, as
    cudaFree is, and the device is waited for before the block can be given out again."""
    p = out(pool, 40 * MB)
    pool.fake_capture(1)
    before = pool.fake_waits()
    assert pool.nspb_free(p) == 0
    assert pool.fake_waits() > before
    assert not pool.fake_capture_ends()
    pool.fake_capture(0)


def test_a_global_capture_refuses(pool):
    p = out(pool, 40 * MB)
    pool.fake_capture(2)
    assert pool.nspb_free(p) != 0
    pool.fake_capture(0)
    assert pool.nspb_free(p) == 0


@pytest.mark.parametrize("kind", ["fake_scratch", "fake_device", "fake_alloc_out"])
def test_kept_blocks_leave_when_memory_is_short(pool, kind):
    """Scratch, a plan's arrays and outputs get the memory of the kept blocks before
    an allocation fails; past that it still fails."""
    pool.fake_capacity(1600 * MB)
    ps = [out(pool, 30 * MB) for _ in range(3)]
    for p in ps:
        assert pool.nspb_free(p) == 0
    assert 90 * MB <= pool.fake_used() <= 90 * MB + 512  # and the block that waits
    p = C.c_void_p()
    assert getattr(pool, kind)(C.byref(p), 1550 * MB) == 0
    assert pool.fake_used() == 1550 * MB
    q = C.c_void_p()
    assert getattr(pool, kind)(C.byref(q), 100 * MB) != 0
    assert pool.nspb_free(p) == 0


HOST_MEMORY = """
import ctypes as C, sys
lib = C.CDLL(sys.argv[1])
lib.nspb_free.argtypes = [C.c_void_p]
lib.fake_alloc_out.argtypes = [C.POINTER(C.c_void_p), C.c_size_t]
lib.fake_used.restype = C.c_size_t
step, p = sys.argv[2], C.c_void_p()
if step == "first":
    lib.fake_no_host_memory(1)
assert lib.fake_alloc_out(C.byref(p), 40 << 20) == 0
if step == "again":
    assert lib.nspb_free(p) == 0
    lib.fake_no_host_memory(1)
    q = C.c_void_p()
    assert lib.fake_alloc_out(C.byref(q), 40 << 20) == 0 and q.value == p.value
if step == "free":
    lib.fake_no_host_memory(1)
assert lib.nspb_free(p) == 0
lib.fake_no_host_memory(0)
assert lib.nspb_trim() == 0
assert lib.fake_used() == 0
"""


@pytest.mark.parametrize("step", ["first", "again", "free"])
def test_no_host_memory_for_the_books(built, step):
    """An exception of the containers stays inside: the call works, the block is not kept."""
    subprocess.run([sys.executable, "-c", HOST_MEMORY, built, step], check=True)


def test_the_wait_keeps_a_block(pool):
    """nspb_free waits by freeing a small block; another one stays allocated meanwhile."""
    for _ in range(3):
        p = out(pool, 40 * MB)
        assert pool.nspb_free(p) == 0
        assert pool.fake_used() == 40 * MB + 512
