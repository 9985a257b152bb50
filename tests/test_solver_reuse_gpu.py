"""One solver workspace over operands that come and go, from several threads, and under a replayed capture."""
import threading

import numpy as np
import pytest
import torch

from gpu_util import dev, host
from plamatrix_b200 import sparse as S

pytestmark = pytest.mark.gpu

ROW1 = 512 * 148  # rows a chip of 148 SMs takes one to a thread


def _banded(n, reach, seed):
    """A symmetric band of `reach` on each side, its diagonal twice the absolute sum of the rest: condition
    number below 30."""
    rng = np.random.default_rng(seed)
    i = np.concatenate([np.arange(n - d) for d in range(1, reach + 1)])
    j = np.concatenate([np.arange(d, n) for d in range(1, reach + 1)])
    v = rng.uniform(-1.0, 1.0, len(i))
    weight = np.bincount(i, np.abs(v), n) + np.bincount(j, np.abs(v), n)
    r, c = np.concatenate([np.arange(n), i, j]), np.concatenate([np.arange(n), j, i])
    v = np.concatenate([2.0 * weight + 1.0, v, v])
    order = np.lexsort((c, r))
    offsets = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(r, minlength=n), out=offsets[1:])
    return offsets, c[order], v[order]


def test_operands_in_the_same_place(checkers):
    """An operand is dropped and another is made over the same values, solution and block buffers, with more
    and with fewer nonzeros: its solve is its own (FP32, blocks of six, more rows than one launch holds)."""
    n = 96_000
    rng = np.random.default_rng(1)
    matrices = [_banded(n, reach, reach) for reach in (1, 3, 2)]
    buffer = torch.empty(max(len(m[1]) for m in matrices), dtype=torch.float32, device="cuda")
    solution = torch.empty(n, dtype=torch.float32, device="cuda")
    inverse = torch.empty(6 * n, dtype=torch.float32, device="cuda")
    b = rng.uniform(-1.0, 1.0, n).astype(np.float32)
    ws = S.IterativeSolverWorkspace()
    options = S.IterativeSolverOptions(relative_tolerance=1e-6)
    for _ in range(3):
        for ro, ci, v in matrices:
            v = v.astype(np.float32)
            buffer[:len(v)] = dev(v)
            diagonal = v[np.repeat(np.arange(n), np.diff(ro)) == ci]
            inverse.copy_(dev((np.eye(6)[None] / diagonal.reshape(-1, 6, 1)).reshape(-1).astype(np.float32)))
            op = S.CsrOperand(S.CSRMatrix(n, n, dev(ro), dev(ci), buffer[:len(v)]))
            solution.zero_()
            report = S.block_pcg(op, dev(b), solution, inverse, 6, ws, options)
            assert report["converged"]
            want, _ = checkers.pcg(ro, ci, v.astype(np.float64), b.astype(np.float64), relative_tolerance=1e-12)
            assert np.linalg.norm(host(solution) - want) <= 1e-4 * np.linalg.norm(want)
            del op


@pytest.mark.parametrize("sizes", [(4 * ROW1 + 777, 8 * ROW1), (3000, ROW1 - 5), (2 * ROW1 + 40, 4 * ROW1 - 3)])
def test_two_sizes_of_one_kernel_at_once(sizes):
    """Two threads solve systems that take the same kernel with different shared memory, each with its own
    workspace and stream: every solve runs and gives the bits of one alone."""
    ops, rhs, want = [], [], []
    for n in sizes:
        ro, ci, v = _banded(n, 2, n)
        ops.append(S.CsrOperand(S.CSRMatrix(n, n, dev(ro), dev(ci), dev(v))))
        rhs.append(torch.linspace(-1.0, 1.0, n, dtype=torch.float64, device="cuda"))
        want.append(torch.zeros_like(rhs[-1]))
        S.pcg(ops[-1], rhs[-1], want[-1])
    torch.cuda.synchronize()
    got, failures = [[], []], []

    def solve(k):
        try:
            stream, ws = torch.cuda.Stream(), S.IterativeSolverWorkspace()
            with torch.cuda.stream(stream):
                for _ in range(40):
                    x = torch.zeros_like(rhs[k])
                    S.pcg(ops[k], rhs[k], x, ws, stream=stream)
                    got[k].append(x)
            stream.synchronize()
            ws.close()
        except Exception as error:  # a thread's exception would be lost
            failures.append(error)

    threads = [threading.Thread(target=solve, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures
    assert all(len(got[k]) == 40 and all(torch.equal(x, want[k]) for x in got[k]) for k in range(2))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("n", [3000, 2 * ROW1, 5 * ROW1])
def test_replayed_capture(dtype, n):
    """A fixed-iteration solve captured once: every replay gives the bits of a direct call, also between
    direct calls with the same workspace."""
    ro, ci, v = _banded(n, 2, n)
    op = S.CsrOperand(S.CSRMatrix(n, n, dev(ro), dev(ci), dev(v, dtype)))
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    sides = [torch.rand(n, generator=g, device="cuda", dtype=torch.float64).to(dtype) - 0.5 for _ in range(6)]
    b, x = torch.empty_like(sides[0]), torch.empty_like(sides[0])
    stream, ws = torch.cuda.Stream(), S.IterativeSolverWorkspace()
    held = []

    def solve(target):
        target.zero_()
        held.append(S.pcg_fixed_iterations_async(op, b, target, 25, ws, stream=stream))

    torch.cuda.synchronize()
    want = []
    with torch.cuda.stream(stream):
        for side in sides:  # one after the other: also the workspace's first growth
            b.copy_(side)
            y = torch.empty_like(b)
            solve(y)
            stream.synchronize()
            want.append(y)
        assert not torch.equal(want[0], want[1])
        graph = torch.cuda.CUDAGraph()
        graph.capture_begin(capture_error_mode="relaxed")
        solve(x)
        graph.capture_end()
        for _ in range(3):
            for k, side in enumerate(sides):
                b.copy_(side)
                graph.replay()
                if k % 3 == 1:
                    y = torch.empty_like(b)
                    solve(y)
                    stream.synchronize()
                    assert torch.equal(y, want[k])
                stream.synchronize()
                assert torch.equal(x, want[k])
    stream.synchronize()
    del graph
    held.clear()
    # nothing of the captured event is left over for the next call
    S.pcg(op, sides[0], torch.zeros_like(x))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_workspace_of_a_large_solve(dtype):
    """Six vectors and small arrays (partial sums and mailboxes, below 4 MB), with the residual kept on the chip
    and as kernels."""
    runtime = pytest.importorskip("cuda.bindings.runtime")
    size = torch.finfo(dtype).bits // 8
    for n in (400_000, 5_000_000):
        offsets, diagonal = torch.arange(n + 1, device="cuda"), torch.arange(n, device="cuda")
        op = S.CsrOperand(S.CSRMatrix(n, n, offsets, diagonal, torch.full((n,), 2.0, dtype=dtype, device="cuda")))
        b, x = torch.ones(n, dtype=dtype, device="cuda"), torch.zeros(n, dtype=dtype, device="cuda")
        torch.cuda.synchronize()
        _, pool = runtime.cudaDeviceGetDefaultMemPool(0)
        used = runtime.cudaMemPoolAttr.cudaMemPoolAttrUsedMemCurrent
        before = int(runtime.cudaMemPoolGetAttribute(pool, used)[1])
        ws = S.IterativeSolverWorkspace()
        assert S.pcg(op, b, x, ws)["converged"]
        after = int(runtime.cudaMemPoolGetAttribute(pool, used)[1])
        assert 0 < after - before <= 6 * n * size + (4 << 20)
        ws.close()
