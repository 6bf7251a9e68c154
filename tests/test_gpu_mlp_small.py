"""Predictions of a few rows, which one host thread converts in parts of 32: at the
edges of the parts, and of the calls that take a batch or more, every row's output is
what the row gives alone, bit for bit, and a NaN in any column is in its row only.
"""
import numpy as np
import pytest

from test_gpu_mlp import fp, lib
from test_gpu_mlp_rows import create

pytestmark = pytest.mark.gpu


def predict(h, x):
    y = np.zeros(len(x), np.float32)
    assert lib().lcmc_mlp_predict(h, fp(np.ascontiguousarray(x)), len(x), fp(y)) == 0
    return y


@pytest.mark.parametrize("n_in,bmax", [(4097, 512), (133, 128), (15, 128)])
def test_rows_alone_and_together(n_in, bmax):
    rng = np.random.default_rng(n_in)
    x = rng.normal(size=(300, n_in)).astype(np.float32)
    h = create(n_in, bmax)
    try:
        alone = np.concatenate([predict(h, x[r:r + 1]) for r in range(len(x))])
        for n in (1, 2, 31, 32, 33, 63, 64, 65, 96, 97, 127, 128, 129, 255, 256, 257, 300):
            np.testing.assert_array_equal(predict(h, x[:n]), alone[:n])
        for col in sorted({0, 3, 7, 8, n_in // 2, n_in - 2, n_in - 1}):
            z = x[:70].copy()
            z[40, col] = np.nan
            y = predict(h, z)
            assert np.isnan(y[40]) and np.array_equal(np.delete(y, 40), np.delete(alone[:70], 40))
    finally:
        lib().lcmc_mlp_destroy(h)
