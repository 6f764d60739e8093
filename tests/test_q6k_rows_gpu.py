"""Q6_K matrices of many rows times two to eight activation rows, against the oracle: edges of its tiles of sixteen rows, of its steps of eight
blocks and of its activation rows; the first and the last two shapes are one activation row, one row and one activation row
behind what it takes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

Q6_K, PATH_GEMV = 14, 1


@pytest.fixture(scope="module")
def ops(mk):
    import importlib
    return importlib.import_module(mk.__name__ + ".ops")


@pytest.mark.parametrize("T,rows,cols", [(1, 2368, 2048), (2, 2368, 256), (8, 2369, 2048), (3, 2383, 2304), (7, 4736, 1792), (5, 2400, 4096), (8, 6000, 4352), (4, 32000, 2048),
                                         (2, 2367, 2048), (9, 2384, 2048)])
def test_rows_match_the_oracle(ops, orc, T, rows, cols):
    w = ops.seed_tensor(0, T, 0.02, Q6_K, rows, cols)
    rng = np.random.default_rng(rows + T)
    x = rng.standard_normal((T, cols)).astype(np.float32)
    x[T - 1, :256] = 0.0        # a block without a scale
    x[0, 256 % cols:] *= 30.0
    got = ops.qmatmul(Q6_K, w, rows, cols, x, PATH_GEMV)
    want = orc.qmatmul(Q6_K, w, rows, cols, x, 1)
    # blocks are integer sums times two factors, the same bits on both sides; K/256 of them are added in another order: 43 roundings at most here,
    # of partial sums that stay below 4 times the largest result
    for t in range(T):
        assert np.max(np.abs(got[t] - want[t])) <= 2e-5 * max(np.max(np.abs(want[t])), 1e-6)
