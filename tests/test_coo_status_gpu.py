"""The status of an asynchronous conversion whose output is refused."""
import ctypes as C

import pytest
import torch

from plamatrix_b200 import _native as N
from plamatrix_b200 import sparse as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nnz, missing", [(3, 0), (3, 1), (3, 2), (-1, None)])
def test_refused_output_leaves_the_count(nnz, missing):
    """The triplets are counted before the output is looked at: the status says how many entries they make."""
    r = torch.tensor([0, 1, 1, 0], device="cuda")
    c = torch.tensor([2, 0, 0, 1], device="cuda")
    v = torch.ones(4, dtype=torch.float64, device="cuda")
    out = [torch.zeros(8, dtype=t, device="cuda") for t in (torch.int64, torch.int64, torch.float64)]
    pointers = [C.c_void_p(None if k == missing else t.data_ptr()) for k, t in enumerate(out)]
    ws = S.SparseOpsWorkspace()
    with pytest.raises(N.InvalidArgument):
        N.call("pm_coo_to_csr_async_f64", ws.handle, S._stream_handle(None), 2, 3, 4, S._ptr(r), S._ptr(c), S._ptr(v),
               nnz, *pointers)
    torch.cuda.synchronize()
    assert ws.check_status() == 3
