"""COO -> CSR of more triplets than one scatter window, in orders that let a group of them skip the windows:
byte for byte against the oracle."""
import numpy as np
import pytest

from gpu_util import dev
from plamatrix_b200 import sparse as S

pytestmark = pytest.mark.gpu


def _order(name, rows, rng):
    count = len(rows)
    if name == "rows":
        return np.argsort(rows, kind="stable")
    if name == "backwards":
        return np.argsort(rows, kind="stable")[::-1]
    if name == "near":  # rows within 1,000 of their place
        return np.argsort(rows + rng.integers(0, 1000, count), kind="stable")
    if name == "two ends":  # every group touches the first and the last window only
        order = np.argsort(rows, kind="stable")
        return np.stack([order[:count // 2], order[count - count // 2:][::-1]], 1).reshape(-1)
    order = np.argsort(rows, kind="stable")  # half in order, half shuffled, in turns of 5,000
    mixed = order.copy()
    mixed[count // 2:] = rng.permutation(order[count // 2:])
    pieces = [mixed[k:k + 5000] for k in range(0, count, 5000)]
    return np.concatenate(pieces[::2] + pieces[1::2])


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("order", ["rows", "backwards", "near", "two ends", "mixed"])
@pytest.mark.parametrize("count", [(1 << 22) + 2, 3 * (1 << 22) + 1022])
def test_orders(checkers, dtype, order, count):
    """Two windows and a few triplets more, and four."""
    rng = np.random.default_rng(count)
    rows, cols = count // 7, 50_000
    r = rng.integers(0, rows, count)
    r = np.ascontiguousarray(r[_order(order, r, rng)])
    if len(r) < count:
        r = np.concatenate([r, r[:count - len(r)]])
    c, v = rng.integers(0, cols, count), rng.standard_normal(count).astype(dtype)
    ro, ci, vv = checkers.coo_to_csr(rows, cols, r, c, v)
    got = S.coo_to_csr(rows, cols, dev(r), dev(c), dev(v)).cpu()
    assert np.array_equal(got[0], ro) and np.array_equal(got[1], ci)
    assert got[2].tobytes() == vv.tobytes()
