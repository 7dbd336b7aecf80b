"""Products of a few dozen activation rows."""
import numpy as np
import pytest

from helpers import ALL

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ex():
    from llama_rust_b200 import Executor
    with Executor(0) as e:
        yield e


def _product(ex, m, x):
    y = np.empty((len(x), m.rows), np.float32)
    ex.gemm_resident(m, len(x), x, y)
    return y


def _same_bits(a, b):
    return np.array_equal(np.ascontiguousarray(a).view(np.uint32), np.ascontiguousarray(b).view(np.uint32))


@pytest.mark.parametrize("rows,cols", [(1, 8), (31, 264), (65, 1032), (9500, 512)])  # ends of tiles, of column steps; four and two weight rows per warp
@pytest.mark.parametrize("name", ["F32", "F16", "BF16"])
def test_rows_of_unpacked_formats_alone_and_in_a_batch(ex, name, rows, cols):
    """Up to 32 activation rows a row's bits do not depend on the batch; above, every sum stays within the bound of a sum of
    `cols` products formed in any order."""
    from llama_rust_b200 import synth
    ex.set_path(0)
    m = ex.synth(ALL[name], rows, cols, 5)
    x = synth.activations(40 * cols, 6).reshape(40, cols)
    alone = np.concatenate([_product(ex, m, x[t:t + 1]) for t in range(32)])
    for n in (3, 4, 5, 8, 9, 16, 17, 32):
        assert _same_bits(_product(ex, m, x[:n]), alone[:n]), n
    w = ex.dequant_rows(m).astype(np.float64)
    exact, size = x.astype(np.float64) @ w.T, np.abs(x).astype(np.float64) @ np.abs(w).T
    for n in (33, 40):
        assert np.all(np.abs(_product(ex, m, x[:n]) - exact[:n]) <= 2.0 ** -24 * (cols + 3) * size[:n]), n
    m.free()
