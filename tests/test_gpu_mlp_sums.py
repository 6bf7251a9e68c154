"""The sums over a batch in the surrogate's backward pass (loss, gradients of b1,
b2, w3, b3): each call's own, whatever the call before it left, for batches that
fill their tile of 128 rows and that do not.

Loss and gradient of b3 are sums of n terms that the outputs give in FP32 exactly
as the kernel forms them; any order of n - 1 additions is within (n - 1) u of the
sum of their magnitudes (u = 2^-24), and the comparison value rounds once more.
The gradients of b1, b2 and w3 are compared with the FP64 oracle: BF16 rounding of
the backward pass is about 1e-2 of them, a sum that kept another call's would be
off by as much as itself.
"""
import ctypes as C

import numpy as np
import pytest

import mlp_oracle as mo
from test_gpu_mlp import fp, lib
from test_gpu_mlp_rows import create

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_in,sizes", [(200, (256, 1, 128, 129, 255)), (4097, (512, 100, 512))])
def test_batch_sums_are_each_calls_own(n_in, sizes):
    L, H = lib(), 128
    k1 = (n_in + 127) // 128 * 128
    o2 = H * k1 + H + H * H
    sections = {"b1": slice(H * k1, H * k1 + H), "b2": slice(o2, o2 + H), "w3": slice(o2 + H, o2 + 2 * H)}
    rng = np.random.default_rng(n_in)
    h = create(n_in, 512)
    try:
        w = np.zeros(L.lcmc_mlp_num_params(h), np.float32)
        assert L.lcmc_mlp_get_params(h, fp(w)) == 0
        for n in sizes:
            x = rng.normal(size=(n, n_in)).astype(np.float32)
            t = (rng.normal(size=n) + 2.0).astype(np.float32)
            g, y, loss = np.zeros_like(w), np.zeros(n, np.float32), C.c_float()
            assert L.lcmc_mlp_gradients(h, fp(x), fp(t), n, fp(g), C.byref(loss)) == 0
            assert L.lcmc_mlp_predict(h, fp(x), n, fp(y)) == 0
            e = y - t
            for got, terms in ((g[-1], np.float32(2) * e / np.float32(n)), (loss.value, e * e / np.float32(n))):
                exact = terms.astype(np.float64)
                assert abs(got - exact.sum()) <= n * 2.0**-24 * np.abs(exact).sum()
            want, _ = mo.gradients(w, x, t.astype(np.float64), n_in)
            for name, s in sections.items():
                assert np.linalg.norm(g[s] - want[s]) < 2e-2 * np.linalg.norm(want[s]), name
    finally:
        L.lcmc_mlp_destroy(h)
