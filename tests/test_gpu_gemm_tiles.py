"""The tensor-core multiply at the edges of its tiles: rows and tokens around 8, 16, 32 and 64, one K stage and several."""
import numpy as np
import pytest

import helpers as H
from brisk_llm_b200 import engine, formats as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", (F.Q4_0, F.Q8_0), ids=lambda f: F.NAMES[f])
@pytest.mark.parametrize("rows,cols", [(1, 128), (31, 384), (65, 128), (129, 1152), (4097, 256)])
def test_tiles(fmt, rows, cols):
    wb, _ = H.random_matrix(fmt, rows, cols, seed=rows)
    x = np.random.default_rng(cols).standard_normal((129, cols)).astype(np.float32)
    want = H.oracle_matmul(fmt, wb, rows, cols, x)
    for n in (2, 15, 17, 33, 64, 65, 129):
        assert np.array_equal(engine.matmul(fmt, wb, rows, cols, x[:n]), want[:n]), n


@pytest.mark.parametrize("fmt", (F.Q4_K, F.Q5_K, F.Q6_K, F.TQ2_0), ids=lambda f: F.NAMES[f])
@pytest.mark.parametrize("rows,cols", [(1, 256), (127, 512), (129, 2304), (4100, 1024)])
def test_super_block_tiles(fmt, rows, cols):
    wb, _ = H.random_matrix(fmt, rows, cols, seed=rows)
    x = np.random.default_rng(cols).standard_normal((129, cols)).astype(np.float32)
    x[3] = 1.0  # equal values: sums of 16 and 32 at their largest
    x[4] = -1.0
    want = H.oracle_matmul(fmt, wb, rows, cols, x)
    for n in (2, 8, 9, 16, 17, 65, 129):
        assert np.array_equal(engine.matmul(fmt, wb, rows, cols, x[:n]), want[:n]), n
