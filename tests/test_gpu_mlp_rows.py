"""How the surrogate's feature rows reach the device, and the training's batches.

* rows are rounded to BF16 on the host (to nearest even): the network gives bit
  for bit what it gives for rows that were rounded before;
* several epochs gather their batches from rows kept on the device: replayed
  from the shuffle's generator with one gradient call per batch and Adam in
  numpy.  A wrong row in a batch changes every weight by about the learning
  rate, 1e-3 against weights of 0.02; a difference in rounding moves only weights
  whose gradient is nearly zero, so the 2-norms are asked to agree to 1e-3.
"""
import ctypes as C

import numpy as np
import pytest
import torch

import oracle_ctypes as oc
from test_gpu_mlp import fp, lib

pytestmark = pytest.mark.gpu


def create(n_in, bmax, seed=5):
    h = C.c_void_p()
    assert lib().lcmc_mlp_create(n_in, 128, bmax, seed, C.byref(h)) == 0
    return h


@pytest.mark.parametrize("n_in,n,bmax", [(4097, 1, 512), (4097, 1111, 512), (133, 700, 128), (128, 4000, 300)])
def test_rows_round_to_nearest_even(n_in, n, bmax):
    rng = np.random.default_rng(n)
    bits = rng.integers(0, 2**32, size=(n, n_in), dtype=np.uint64).astype(np.uint32)
    bits = (bits & np.uint32(0x83FFFFFF)) | np.uint32(0x3C000000)  # magnitudes 2^-7 .. 2
    ties = rng.random(size=(n, n_in)) < 0.3
    bits[ties] = (bits[ties] & np.uint32(0xFFFF0000)) | np.uint32(0x8000)
    x = bits.view(np.float32)
    rounded = torch.from_numpy(x).bfloat16().float().numpy()
    assert not np.array_equal(x, rounded)
    h = create(n_in, bmax)
    try:
        a, b = np.zeros(n, np.float32), np.zeros(n, np.float32)
        assert lib().lcmc_mlp_predict(h, fp(x), n, fp(a)) == 0
        assert lib().lcmc_mlp_predict(h, fp(rounded), n, fp(b)) == 0
        np.testing.assert_array_equal(a, b)
        x[n // 2, n_in - 1] = np.nan  # only its own row
        assert lib().lcmc_mlp_predict(h, fp(x), n, fp(b)) == 0
        assert np.isnan(b[n // 2])
        keep = np.arange(n) != n // 2
        np.testing.assert_array_equal(a[keep], b[keep])
    finally:
        lib().lcmc_mlp_destroy(h)


def shuffles(n, seed, epochs):
    idx = np.arange(n)
    key = [seed & 0xFFFFFFFF, seed >> 32]
    for ep in range(epochs):
        for i in range(n - 1, 0, -1):
            j = oc.philox([i, ep, 0, 0x301], key)[0] % (i + 1)
            idx[i], idx[j] = idx[j], idx[i]
        yield idx.copy()


@pytest.mark.parametrize("n,batch,epochs", [(330, 100, 3), (512, 256, 2), (200, 200, 2)])
def test_epochs_take_the_shuffled_rows(n, batch, epochs):
    n_in, seed, lr = 200, 7, np.float32(1e-3)
    rng = np.random.default_rng(batch)
    x = rng.normal(size=(n, n_in)).astype(np.float32)
    t = (x[:, :40].sum(1) + 3.0).astype(np.float32)
    a, b = create(n_in, 256), create(n_in, 256)
    L = lib()
    L.lcmc_mlp_set_params.argtypes = [C.c_void_p, C.POINTER(C.c_float)]
    try:
        loss = C.c_float()
        assert L.lcmc_mlp_train(a, fp(x), fp(t), n, epochs, batch, lr, seed, C.byref(loss)) == 0
        w = np.zeros(L.lcmc_mlp_num_params(b), np.float32)
        got = np.zeros_like(w)
        assert L.lcmc_mlp_get_params(a, fp(got)) == 0
        assert L.lcmc_mlp_get_params(b, fp(w)) == 0
        start = w.copy()
        g, m, v, step = np.zeros_like(w), np.zeros_like(w), np.zeros_like(w), 0
        for idx in shuffles(n, seed, epochs):
            losses = []
            for off in range(0, n - batch + 1, batch):
                rows = idx[off:off + batch]
                l = C.c_float()
                bx, bt = np.ascontiguousarray(x[rows]), np.ascontiguousarray(t[rows])
                assert L.lcmc_mlp_gradients(b, fp(bx), fp(bt), batch, fp(g), C.byref(l)) == 0
                losses.append(l.value)
                step += 1
                m = np.float32(0.9) * m + np.float32(0.1) * g
                v = np.float32(0.999) * v + np.float32(0.001) * g * g
                w = w - lr * (m / np.float32(1 - 0.9**step)) / (np.sqrt(v / np.float32(1 - 0.999**step)) + np.float32(1e-8))
                assert L.lcmc_mlp_set_params(b, fp(w)) == 0
        assert loss.value == pytest.approx(np.mean(losses), rel=1e-3)
        assert np.linalg.norm(got - w) < 1e-3 * np.linalg.norm(w)
        assert np.linalg.norm(got - start) > 0.02 * np.linalg.norm(w)
    finally:
        L.lcmc_mlp_destroy(a)
        L.lcmc_mlp_destroy(b)
