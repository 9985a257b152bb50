"""CSR operands of more nonzeros than the bytes of one array fit in an int.

Tolerance: the summation-order bound (row length + 1) eps sum |a_ij x_j|."""
import pytest
import torch

from plamatrix_b200 import sparse as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype, nonzeros", [(torch.float64, 1 << 28), (torch.float32, 1 << 29)])
def test_spmv_of_many_nonzeros(dtype, nonzeros):
    """Eight nonzeros in every row: from 2^28 FP64 (2^29 FP32) values on, an array is 2 GB or more."""
    rows, cols, width = nonzeros // 8 + 1003, 1 << 16, 8
    g = torch.Generator(device="cuda")
    g.manual_seed(11)
    first = torch.randint(0, cols, (rows,), generator=g, device="cuda")
    columns = torch.empty((rows, width), dtype=torch.int64, device="cuda")
    for k in range(width):
        columns[:, k] = (first + 7919 * k) % cols
    values = torch.rand((rows, width), generator=g, device="cuda", dtype=dtype) + 0.5
    x = torch.rand(cols, generator=g, device="cuda", dtype=dtype) + 0.5
    offsets = torch.arange(rows + 1, device="cuda") * width
    op = S.CsrOperand(S.CSRMatrix(rows, cols, offsets, columns.view(-1), values.view(-1)))
    y = op.spmv(x)
    for lo in range(0, rows, 1 << 22):  # every entry is positive: the sum is the bound's size too
        part = slice(lo, min(rows, lo + (1 << 22)))
        want = (values[part].double() * x.double()[columns[part]]).sum(1)
        bound = (width + 1) * torch.finfo(dtype).eps * want
        assert bool(((y[part].double() - want).abs() <= bound).all())
