"""COO -> CSR where its kernels change: rows of 0 to 17 entries (the register networks of 8, 12 and 16,
the long rows from 17), runs of 32 rows that fill or exceed their staged tile, last tiles of every
length, and inputs at the edges of the scatter windows.  Byte for byte against the oracle."""
import numpy as np
import pytest
import torch

from gpu_util import dev, host, tdtype
from plamatrix_b200 import _native as N
from plamatrix_b200 import sparse as S

pytestmark = pytest.mark.gpu


def _compare(checkers, rows, cols, r, c, v):
    ro, ci, vv = checkers.coo_to_csr(rows, cols, r, c, v)
    out = S.coo_to_csr(rows, cols, dev(r), dev(c), dev(v))
    got = out.cpu()
    assert np.array_equal(got[0], ro) and np.array_equal(got[1], ci)
    assert got[2].tobytes() == vv.tobytes()
    again = S.CSRMatrix.empty(rows, cols, len(ci), tdtype(v.dtype))
    ws = S.SparseOpsWorkspace()
    S.coo_to_csr_async(rows, cols, dev(r), dev(c), dev(v), again, ws)
    torch.cuda.synchronize()
    assert ws.check_status() == len(ci)
    assert np.array_equal(host(again.row_offsets), ro) and host(again.values).tobytes() == vv.tobytes()


def _rows_of(lengths, cols, seed, dtype):
    rng = np.random.default_rng(seed)
    r = np.repeat(np.arange(len(lengths)), lengths)
    c = rng.integers(0, cols, len(r))
    order = rng.permutation(len(r))
    return r[order].astype(np.int64), c[order].astype(np.int64), rng.standard_normal(len(r)).astype(dtype)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("rows", [1, 31, 32, 33, 255, 257, 1000])
@pytest.mark.parametrize("most", [1, 8, 9, 12, 13, 16, 17])
def test_row_lengths(checkers, dtype, rows, most):
    """Mixed lengths up to `most`; few columns, so that most rows have duplicates."""
    rng = np.random.default_rng(rows * 100 + most)
    lengths = rng.integers(0, most + 1, rows)
    lengths[rows // 2] = most
    _compare(checkers, rows, 11, *_rows_of(lengths, 11, most, dtype))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("length, extra", [(12, 0), (12, 1), (16, 0), (16, 1), (7, 2500)])
def test_tiles_at_their_capacity(checkers, dtype, length, extra):
    """32 rows of twelve entries fill a tile; one more entry, or a long row among them, goes past it."""
    lengths = np.full(96, length)
    lengths[40] += extra
    _compare(checkers, 96, 1 << 20, *_rows_of(lengths, 1 << 20, length + extra, dtype))


@pytest.mark.parametrize("count", [(1 << 22) - 1, (1 << 22) + 1, (1 << 23) + 1])
def test_scatter_windows(checkers, count):
    """2^22 records fill the window of one pass."""
    rng = np.random.default_rng(count)
    rows, cols = 600_000, 1_000_000
    r, c = rng.integers(0, rows, count), rng.integers(0, cols, count)
    _compare(checkers, rows, cols, r, c, rng.standard_normal(count))


@pytest.mark.parametrize("count", [100, (1 << 22) + 7])
def test_errors_name_the_lowest_offset(count):
    """A column out of range, a row out of range and a value that is not finite, each also where the
    triplet is another window's."""
    rng = np.random.default_rng(3)
    rows, cols = 5000, 4000
    r, c, v = rng.integers(0, rows, count), rng.integers(0, cols, count), rng.standard_normal(count)
    for bad, where in (("column", count - 3), ("row", count // 2), ("value", 50)):
        r2, c2, v2 = r.copy(), c.copy(), v.copy()
        if bad == "column":
            c2[where], c2[-1] = cols, -1
        elif bad == "row":
            r2[where], r2[-1], c2[-2] = -1, rows, cols
        else:
            v2[where], v2[-1] = np.inf, np.nan
        with pytest.raises(N.PlamatrixError, match=f"source offset {where}$"):
            S.coo_to_csr(rows, cols, dev(r2), dev(c2), dev(v2))
