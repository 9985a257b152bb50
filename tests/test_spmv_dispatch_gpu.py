"""SpMV and the solvers where the choice of a row kernel changes.

Tolerances: SpMV within the summation-order bound (row length + 1) eps sum |a_ij x_j|.  The matrices are
strictly diagonally dominant with a condition number below 30: a solution of an FP64 solve to 1e-10 is within
1e-8 of the reference's, an FP32 one (1e-6, vectors rounded to FP32) within 1e-4."""
import numpy as np
import pytest
import torch

from gpu_util import dev, host, tdtype
from plamatrix_b200 import _native as N
from plamatrix_b200 import sparse as S

pytestmark = pytest.mark.gpu


def _symmetric(lengths, seed):
    """A symmetric matrix whose rows have about `lengths` nonzeros: a diagonal of twice the absolute sum of
    the rest of the row, and wrapped bands whose reach follows the length."""
    rng = np.random.default_rng(seed)
    n = len(lengths)
    reach = (np.asarray(lengths) - 1) // 2
    i = np.repeat(np.arange(n), reach)
    step = np.concatenate([np.arange(1, k + 1) for k in reach]) if len(i) else np.zeros(0, np.int64)
    j = (i + step) % n
    keep = i != j
    i, j = i[keep], j[keep]
    v = rng.uniform(-1.0, 1.0, len(i))
    weight = np.zeros(n)
    np.add.at(weight, i, np.abs(v))
    np.add.at(weight, j, np.abs(v))
    r, c = np.concatenate([np.arange(n), i, j]), np.concatenate([np.arange(n), j, i])
    v = np.concatenate([2.0 * weight + 1.0, v, v])
    order = np.lexsort((c, r))
    offsets = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(r, minlength=n), out=offsets[1:])
    return offsets, c[order].astype(np.int64), v[order]


def _operand(matrix, dtype):
    ro, ci, v = matrix
    n = len(ro) - 1
    return S.CsrOperand(S.CSRMatrix(n, n, dev(ro), dev(ci), dev(v.astype(dtype))))


def _check_product(checkers, matrix, dtype):
    ro, ci, v = matrix
    n = len(ro) - 1
    op = _operand(matrix, dtype)
    x = np.random.default_rng(n).uniform(-1.0, 1.0, n).astype(dtype)
    want = checkers.csr_spmv(ro, ci, v, x.astype(np.float64))
    size = checkers.csr_spmv(ro, ci, np.abs(v), np.abs(x.astype(np.float64)))
    error = np.abs(host(op.spmv(dev(x))).astype(np.float64) - want)
    assert np.all(error <= (np.diff(ro) + 1) * np.finfo(dtype).eps * size)
    return op, x


def _check(checkers, matrix, dtype, solvers=("pcg",)):
    ro, ci, v = matrix
    n = len(ro) - 1
    v = v.astype(dtype).astype(np.float64)
    op, x = _check_product(checkers, (ro, ci, v), dtype)
    solution, report = checkers.pcg(ro, ci, v, x.astype(np.float64), relative_tolerance=1e-12)
    assert report["converged"]
    options = S.IterativeSolverOptions(relative_tolerance=1e-10 if dtype == np.float64 else 1e-6)
    for kind in solvers:
        got = torch.zeros(n, dtype=tdtype(dtype), device="cuda")
        more = ()
        if kind == "block_pcg":  # the inverse diagonal in blocks of three
            inverse = np.zeros((n // 3, 3, 3))
            rows = np.repeat(np.arange(n), np.diff(ro))
            inverse[np.arange(n) // 3, np.arange(n) % 3, np.arange(n) % 3] = 1.0 / v[rows == ci]
            more = (dev(inverse.reshape(-1).astype(dtype)), 3)
        report = getattr(S, kind)(op, dev(x), got, *more, options=options)
        assert report["converged"]
        tolerance = 1e-8 if dtype == np.float64 else 1e-4
        assert np.linalg.norm(host(got) - solution) <= tolerance * np.linalg.norm(solution)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [700, 5000])
@pytest.mark.parametrize("length", [33, 257, 447, 449, 513, 655])
def test_long_rows(checkers, dtype, n, length):
    """Fewer and more than fourteen nonzeros per lane, even and uneven rows, in one launch and as kernels."""
    even = np.full(n, length)
    _check(checkers, _symmetric(even, n), dtype, ("pcg", "cg"))
    uneven = np.random.default_rng(length).integers(length // 2, length + length // 2, n)
    _check(checkers, _symmetric(uneven, n), dtype)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("rows", [32, 33, 4800])
@pytest.mark.parametrize("held", [0, 1, 319, 320, 321, 640, 641, 5000])
def test_tiles_of_short_rows(checkers, dtype, rows, held):
    """32 rows of `held` nonzeros among rows of five: a tile below, at and past its capacity of 320, in two
    pieces and in many, starting at every offset from a 16-byte boundary."""
    rng = np.random.default_rng(held)
    for lead in range(4 if rows > 64 else 1):
        lengths = np.full(rows, 5 if rows > 64 else 0)
        first = 64 if rows > 64 else 0
        lengths[0] += lead
        lengths[first:first + 32] = rng.multinomial(held, np.full(32, 1.0 / 32.0))
        if rows <= 64 and held > 8 * rows:
            lengths = np.concatenate([lengths, np.zeros(held // 8 + 1, lengths.dtype)])  # a mean of at most eight
        offsets = np.zeros(len(lengths) + 1, np.int64)
        np.cumsum(lengths, out=offsets[1:])
        columns = rng.integers(0, len(lengths), offsets[-1])
        values = rng.standard_normal(offsets[-1]).astype(dtype).astype(np.float64)
        _check_product(checkers, (offsets, columns, values), dtype)


@pytest.mark.parametrize("longest", [7, 13])
def test_tiles_in_the_iteration_graph(checkers, longest):
    """Block PCG of more rows than one launch holds, FP32: tiles up to and past their capacity."""
    n = 96_000
    rows = np.where(np.arange(n) % 640 < 32, longest, 7)
    _check(checkers, _symmetric(rows, n), np.float32, ("block_pcg",))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [300, 6000])
@pytest.mark.parametrize("longest", [127, 129, 299])
def test_one_long_row(checkers, dtype, n, longest):
    """Short rows and one of up to or more than 128 nonzeros: rows in registers, or staged tiles."""
    lengths = np.full(n, 3)
    lengths[n // 2] = 2 * (longest - 2) + 1  # its diagonal, its reach and the neighbour before it
    matrix = _symmetric(lengths, longest)
    assert np.diff(matrix[0]).max() == longest
    _check(checkers, matrix, dtype, ("pcg", "cg", "block_pcg"))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [700, 5000])
@pytest.mark.parametrize("longest", [100, 270, 600])
def test_one_long_row_among_longer_ones(checkers, dtype, n, longest):
    """Rows of 21 and one of 100 to 600: the lanes of every row read one after the other, or in rounds."""
    lengths = np.full(n, 21)
    lengths[n // 2] = 2 * (longest - 11) + 1
    matrix = _symmetric(lengths, longest)
    assert np.diff(matrix[0]).max() == longest
    _check(checkers, matrix, dtype, ("pcg", "cg"))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("row", [0, 200, 399])
def test_diagonal_near_zero(dtype, row):
    """A diagonal entry far below its row's largest, with all values below one: the row is named.  Long and
    short rows."""
    n = 400
    ro, ci, v = _symmetric(np.where(np.arange(n) % 50 == 0, 41, 5), 3)
    v = v / np.abs(v).max() / 2.0
    at = np.repeat(np.arange(n), np.diff(ro))
    v[(at == row) & (ci == row)] = 4.0 * np.finfo(dtype).eps * np.abs(v[(at == row) & (ci != row)]).max()
    x = torch.zeros(n, dtype=tdtype(dtype), device="cuda")
    with pytest.raises(N.PlamatrixError, match=f"near zero at row {row}$"):
        S.pcg(_operand((ro, ci, v), dtype), torch.ones_like(x), x)
