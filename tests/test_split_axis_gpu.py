"""Reductions that split their axis between blocks, at the sizes where chunks and remainders meet, against numpy (GPU tests)."""
import numpy as np
import pytest

from tests import util

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("shape", [(31, 5), (32, 2), (33, 3), (256, 10), (1000, 625), (4096, 33), (100_003, 7),
                                   (3, 64, 17), (2, 5000, 32), (40, 32, 100)])
def test_reduce_few_columns(fresh, shape, dt):
    e = fresh
    axis = len(shape) - 2
    x = util.normal(311 + shape[-1], shape, dt)
    tx, y = e.tensor(x), e.empty(shape[:axis] + shape[axis + 1:], dt)
    for _ in range(2):                      # twice: the arrival counters must be back at zero
        e.Reduce("sum", tx, y, axis)
        # any order of n additions stays within n * eps of the sum of magnitudes; four chains and a tree
        # need far fewer
        n, eps = shape[axis], np.finfo(dt).eps
        bound = (n // 4 + 16) * eps * np.abs(x).astype(np.float64).sum(axis)
        assert (np.abs(y.numpy() - x.astype(np.float64).sum(axis)) <= bound).all()
        e.Reduce("max", tx, y, axis)
        assert np.array_equal(y.numpy(), x.max(axis))


def test_reduce_few_columns_special_values(fresh):
    e = fresh
    x = np.full((300, 6), -np.inf, np.float32)
    x[:, 1] = np.nan
    x[7, 2] = np.inf
    x[:, 3] = -np.finfo(np.float32).max
    x[250, 4] = np.nan
    x[251, 4] = 2.0
    x[:, 5] = 0.0
    y = e.empty((6,))
    e.Reduce("max", e.tensor(x), y, 0)      # a NaN never wins, as in the thread-per-column walk
    assert np.array_equal(y.numpy(), np.array([-np.inf, -np.inf, np.inf, -np.finfo(np.float32).max, 2.0, 0.0], np.float32))
    e.Reduce("sum", e.tensor(x), y, 0)
    got = y.numpy()
    assert got[0] == -np.inf and np.isnan(got[1]) and got[3] == -np.inf and np.isnan(got[4]) and got[5] == 0.0
