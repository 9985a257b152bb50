"""The one-launch CG / PCG and the staged SpMV at the sizes where their dispatch changes: rows per
thread (1, 2, 4), the kept residual, rows longer than a staged tile, values off a 16-byte boundary,
every SpMV shape, block inverses, and solves on two streams at once.

Tolerances: SpMV within the summation-order bound (row length + 1) eps sum |a_ij x_j|.  A solution of
an FP64 solve to 1e-10 is within 1e-8 of the oracle's (condition number below 100 for these
matrices); FP32 vectors carry a relative error of at most condition x eps32 x sqrt(iterations), below
2e-4."""
import threading

import numpy as np
import pytest
import torch

from gpu_util import dev, host
from plamatrix_b200 import sparse as S

pytestmark = pytest.mark.gpu

SMS = 148
ROW1 = 512 * SMS  # one row per thread up to here, two up to 2x, four up to 4x, then tiles


def _banded(n, dtype, seed, long_row=0):
    """A diagonally dominant symmetric matrix: a band of three on each side with random holes and,
    with `long_row`, a first row and column of that many entries.  Condition number below 100."""
    rng = np.random.default_rng(seed)
    r, c = [], []
    for d in (1, 2, 3):
        i = np.arange(n - d)[rng.random(max(n - d, 0)) < 0.8] if n > d else np.zeros(0, np.int64)
        r.append(i)
        c.append(i + d)
    if long_row:
        j = np.arange(4, min(n, long_row + 4))
        r.append(np.zeros(len(j), np.int64))
        c.append(j)
    r, c = np.concatenate(r).astype(np.int64), np.concatenate(c).astype(np.int64)
    v = rng.uniform(-1.0, 1.0, len(r))
    # entries of the long row are small enough to keep the rows balanced
    v[(r == 0) & (c >= 4)] *= 1e-3
    weight = np.zeros(n)
    np.add.at(weight, r, np.abs(v))
    np.add.at(weight, c, np.abs(v))
    rows = np.concatenate([np.arange(n), r, c])
    cols = np.concatenate([np.arange(n), c, r])
    vals = np.concatenate([weight + rng.uniform(0.1, 1.0, n), v, v])
    order = np.lexsort((cols, rows))
    ro = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(rows, minlength=n), out=ro[1:])
    return ro, cols[order], vals[order].astype(dtype)


def _operand(ro, ci, v, offset=0):
    n = len(ro) - 1
    values = torch.empty(len(v) + offset, dtype=dev(v[:1]).dtype, device="cuda")[offset:]
    values.copy_(dev(v))
    return S.CsrOperand(S.CSRMatrix(n, n, dev(ro), dev(ci), values))


def _check_spmv(checkers, op, ro, ci, v, dtype, seed):
    x = np.random.default_rng(seed).standard_normal(len(ro) - 1).astype(dtype)
    ref = checkers.csr_spmv(ro, ci, v.astype(np.float64), x.astype(np.float64))
    size = checkers.csr_spmv(ro, ci, np.abs(v.astype(np.float64)), np.abs(x.astype(np.float64)))
    y = host(op.spmv(dev(x))).astype(np.float64)
    assert np.all(np.abs(y - ref) <= (np.diff(ro) + 1) * np.finfo(dtype).eps * size + 1e-300)


def _check_solve(checkers, op, ro, ci, v, dtype, kind="pcg", **kw):
    n = len(ro) - 1
    b = np.random.default_rng(n).uniform(-1.0, 1.0, n).astype(dtype)
    tol = 1e-10 if dtype == np.float64 else 1e-6
    x_ref, rep_ref = checkers.pcg(ro, ci, v.astype(np.float64), b.astype(np.float64), relative_tolerance=1e-12)
    x = torch.zeros(n, dtype=op.dtype, device="cuda")
    rep = getattr(S, kind)(op, dev(b), x, options=S.IterativeSolverOptions(relative_tolerance=tol), **kw)
    assert rep["converged"] and rep_ref["converged"]
    error = np.linalg.norm(host(x).astype(np.float64) - x_ref)
    assert error <= (1e-8 if dtype == np.float64 else 2e-4) * np.linalg.norm(x_ref)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [1, 31, 33, 1000, 256 * SMS + 1, ROW1, ROW1 + 1, 2 * ROW1 + 33, 4 * ROW1, 4 * ROW1 + 1])
def test_sizes_at_the_edges_of_the_dispatch(checkers, dtype, n):
    ro, ci, v = _banded(n, dtype, n)
    op = _operand(ro, ci, v)
    _check_spmv(checkers, op, ro, ci, v, dtype, n)
    _check_solve(checkers, op, ro, ci, v, dtype)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [500, ROW1 + 500, 4 * ROW1 + 500])
@pytest.mark.parametrize("long_row, offset", [(300, 0), (0, 1), (1500, 1)])
def test_long_rows_and_unaligned_values(checkers, dtype, n, long_row, offset):
    ro, ci, v = _banded(n, dtype, n + long_row, min(long_row, n - 4))
    op = _operand(ro, ci, v, offset)
    _check_spmv(checkers, op, ro, ci, v, dtype, n)
    _check_solve(checkers, op, ro, ci, v, dtype)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [999, 4 * ROW1 + 40])
@pytest.mark.parametrize("shape", [0, 1, 2, 4, 8, 16, 32])
def test_every_shape_in_one_launch(checkers, dtype, n, shape):
    ro, ci, v = _banded(n, dtype, n)
    op = _operand(ro, ci, v)
    op.set_kernel(shape)
    _check_solve(checkers, op, ro, ci, v, dtype)
    _check_solve(checkers, op, ro, ci, v, dtype, kind="cg")


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [6, 1200, 6 * ROW1])
def test_block_inverses(checkers, dtype, n):
    """Blocks of six: the residual of a block's rows comes from other threads."""
    ro, ci, v = _banded(n, dtype, n)
    blocks = np.zeros((n // 6, 6, 6))
    rows = np.repeat(np.arange(n), np.diff(ro))
    inside = rows // 6 == ci // 6
    blocks[rows[inside] // 6, rows[inside] % 6, ci[inside] % 6] = v[inside]
    inverse = np.ascontiguousarray(np.linalg.inv(blocks).reshape(-1).astype(dtype))
    _check_solve(checkers, _operand(ro, ci, v), ro, ci, v, dtype, kind="block_pcg", inverse_blocks=dev(inverse),
                 block_size=6)


def test_solves_on_two_streams_at_once(checkers):
    """Two threads, each with its own workspace and stream: the same bits as one after the other."""
    systems = [_banded(n, np.float64, n) for n in (3000, 4 * ROW1 + 777)]
    want, ops, rhs = [], [], []
    for ro, ci, v in systems:
        ops.append(_operand(ro, ci, v))
        rhs.append(torch.linspace(-1.0, 1.0, len(ro) - 1, dtype=torch.float64, device="cuda"))
        x = torch.zeros_like(rhs[-1])
        S.pcg(ops[-1], rhs[-1], x)
        want.append(x)
    torch.cuda.synchronize()
    got = [[], []]

    def solve(k):
        stream = torch.cuda.Stream()
        ws = S.IterativeSolverWorkspace()
        for _ in range(10):
            with torch.cuda.stream(stream):
                x = torch.zeros_like(rhs[k])
                S.pcg(ops[k], rhs[k], x, ws, stream=stream)
            stream.synchronize()
            got[k].append(x)
        ws.close()

    threads = [threading.Thread(target=solve, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(2):
        assert len(got[k]) == 10 and all(torch.equal(x, want[k]) for x in got[k])
