"""A two-call numeric step looks at a sample of the B rows that A reads: operands whose nnz
field is larger than their last row pointer, with nothing of use behind the entries."""
import ctypes as C

import numpy as np
import pytest

import nsp_b200 as nb
import oracle
from nsp_b200 import _lib

from conftest import assert_bitwise, assert_same_structure

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [40_000, 9000, 1024])
def test_entries_past_the_last_row_are_not_read(cuda, n):
    import torch
    d = 40 if n == 1024 else 9
    A, B = nb.gen.random(n, 5000, d, d, seed=1), nb.gen.random(5000, 300_000, 3, 9, seed=2)
    dA, dB = A.to_device(), B.to_device()
    extra = 100_000
    # columns of B's last row, which an average would show, inside B all the same
    dA.col = torch.cat([dA.col, torch.full((extra,), 4999, dtype=torch.int32, device="cuda")])
    dA.val = torch.cat([dA.val, torch.full((extra,), float("nan"), dtype=torch.float64, device="cuda")])
    rp, col, val = oracle.spgemm(A, B)
    drp = torch.from_numpy(np.ascontiguousarray(rp, dtype=np.int32)).cuda()
    a, b, c, o = dA.as_in(), dB.as_in(), _lib.CsrOut(), nb.make_opts()
    a.nnz = A.nnz + extra
    dcol = torch.empty(len(col), dtype=torch.int32, device="cuda")
    dval = torch.empty(len(col), dtype=torch.float64, device="cuda")
    c.nrows, c.ncols, c.nnz, c.capacity = n, B.ncols, len(col), len(col)
    c.rowptr, c.col, c.val = drp.data_ptr(), dcol.data_ptr(), dval.data_ptr()
    st = nb.lib.nspb_spgemm_numeric(C.byref(a), C.byref(b), C.byref(c), C.byref(o), None)
    assert st == 0
    assert_same_structure(drp.cpu().numpy(), dcol.cpu().numpy(), rp, col)
    assert_bitwise(dval.cpu().numpy(), val)
