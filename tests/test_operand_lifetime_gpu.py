"""A CSR operand that is dropped while a product with it is still queued: its memory stays until that is done."""
import pytest
import torch

from plamatrix_b200 import sparse as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_operand_dropped_behind_queued_work(dtype):
    """`spmv(matrix, x)` keeps its operand only during the call.  Products of positive numbers are summed
    in storage order: within (row length + 1) eps of the 64-bit sum."""
    rows, width = 1 << 20, 7
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    columns = torch.randint(0, rows, (rows, width), generator=g, device="cuda")
    values = torch.rand((rows, width), generator=g, device="cuda", dtype=dtype) + 0.5
    x = torch.rand(rows, generator=g, device="cuda", dtype=dtype) + 0.5
    matrix = S.CSRMatrix(rows, rows, torch.arange(rows + 1, device="cuda") * width, columns.view(-1), values.view(-1))
    want = (values.double() * x.double()[columns]).sum(1)
    product = torch.randn(4096, 4096, device="cuda")
    for _ in range(4):
        op = S.CsrOperand(matrix)
        y = torch.empty(rows, dtype=dtype, device="cuda")
        for _ in range(10):
            product = product @ product * 1e-3  # the product below waits behind these
        op.spmv(x, y)
        del op
        taken = torch.full((rows * width,), -1, dtype=torch.int32, device="cuda")
        assert bool(((y.double() - want).abs() <= (width + 1) * torch.finfo(dtype).eps * want).all())
        del taken
    y = S.spmv(matrix, x)
    assert bool(((y.double() - want).abs() <= (width + 1) * torch.finfo(dtype).eps * want).all())


def test_operand_dropped_during_a_capture():
    """Another operand with work queued on another stream is dropped while a stream is captured (relaxed mode,
    in which memory may be released): the capture goes on and replays."""
    n = 10_000
    offsets, columns = torch.arange(n + 1, device="cuda"), torch.arange(n, device="cuda")
    values, x = torch.rand(n, dtype=torch.float64, device="cuda"), torch.rand(n, dtype=torch.float64, device="cuda")
    y, z = torch.zeros_like(x), torch.zeros_like(x)
    kept, dropped = (S.CsrOperand(S.CSRMatrix(n, n, offsets, columns, values)) for _ in range(2))
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    dropped.spmv(x, z)
    kept.spmv(x, y)
    torch.cuda.synchronize()
    dropped.spmv(x, z)
    with torch.cuda.stream(stream):
        graph.capture_begin(capture_error_mode="relaxed")
        dropped.spmv(x, z)
        kept.spmv(x, y)
        graph.capture_end()
        graph.reset()
        dropped.spmv(x, z)
        graph = torch.cuda.CUDAGraph()
        graph.capture_begin(capture_error_mode="relaxed")
        kept.spmv(x, y)
        del dropped
        kept.spmv(x, y)
        graph.capture_end()
        y.zero_()
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, values * x) and torch.equal(z, values * x)
