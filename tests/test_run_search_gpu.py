"""When row runs are looked for at all: two calls need larger products than one. Where the
library looks by itself, a call has the launches of one that is told to (row_kernel 8)."""
import pytest

import nsp_b200 as nb
from nsp_b200 import _lib

pytestmark = pytest.mark.gpu

RUNS = 8


def launches(d, e, row_kernel, two):
    """Launches of a product: of the call, or of its symbolic and numeric calls."""
    import ctypes as C
    import torch
    if not two:
        return [nb.spgemm(d, e, row_kernel=row_kernel, return_stats=True)[1]["launches"]]
    o, st = nb.make_opts(row_kernel=row_kernel), _lib.Stats()
    a, b, c = d.as_in(), e.as_in(), _lib.CsrOut()
    rp = torch.empty(d.nrows + 1, dtype=torch.int32, device="cuda")
    c.rowptr = rp.data_ptr()
    out = []
    assert nb.lib.nspb_spgemm_symbolic(C.byref(a), C.byref(b), C.byref(c), C.byref(o), C.byref(st)) == 0
    out.append(st.launches)
    col = torch.empty(c.nnz, dtype=torch.int32, device="cuda")
    val = torch.empty(c.nnz, dtype=torch.float64, device="cuda")
    c.col, c.val, c.capacity = col.data_ptr(), val.data_ptr(), c.nnz
    assert nb.lib.nspb_spgemm_numeric(C.byref(a), C.byref(b), C.byref(c), C.byref(o), C.byref(st)) == 0
    out.append(st.launches)
    return out


# 7-point: 47 products a row; 27-point: about 660
@pytest.mark.parametrize("npts,dims,one,two", [
    (7, (50, 50, 50), False, False), (7, (60, 60, 60), True, False), (7, (72, 72, 72), True, True),
    (27, (30, 30, 30), False, False), (27, (36, 36, 36), True, False), (27, (42, 42, 42), True, True)])
def test_size_rule(cuda, npts, dims, one, two):
    d = nb.gen.stencil(*dims, npts=npts).to_device()
    for calls, wanted in ((False, one), (True, two)):
        auto, told = launches(d, d, 0, calls), launches(d, d, RUNS, calls)
        assert [x == y for x, y in zip(auto, told)] == [wanted] * len(auto), (auto, told)
