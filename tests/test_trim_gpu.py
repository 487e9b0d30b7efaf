"""nb.trim(): a Python program gets the memory of freed outputs back for its other allocators."""
import pytest

import nsp_b200 as nb

pytestmark = pytest.mark.gpu


def test_trim_gives_memory_to_other_allocators(cuda):
    import torch
    A = nb.gen.stencil(64, npts=27).to_device()
    nb.trim()
    C = nb.spgemm(A, A)
    nbytes = 12 * int(C.nnz)
    del C
    torch.cuda.synchronize()
    kept = torch.cuda.mem_get_info()[0]
    nb.trim()
    assert torch.cuda.mem_get_info()[0] - kept >= nbytes - (4 << 20)
    nb.trim()  # nothing kept: nothing happens
