"""Networks used from several threads at once, each with its own row threads: small
and large calls in turn give what they give alone, bit for bit, and networks come
and go while others work.
"""
import threading

import numpy as np
import pytest

from test_gpu_mlp import fp, lib
from test_gpu_mlp_rows import create
from test_gpu_mlp_small import predict

pytestmark = pytest.mark.gpu


def test_networks_in_threads():
    n_in = 4097
    rng = np.random.default_rng(11)
    x = rng.normal(size=(1500, n_in)).astype(np.float32)
    h = create(n_in, 256)
    want = predict(h, x)
    lib().lcmc_mlp_destroy(h)
    failed = []

    def work(seed):
        r = np.random.default_rng(seed)
        try:
            for _ in range(4):
                h = create(n_in, 256)
                for n in (*r.integers(1, 1500, size=8), 1500, 1, 700):
                    o = int(r.integers(0, 1501 - n))
                    if not np.array_equal(predict(h, x[o:o + n]), want[o:o + n]):
                        failed.append((seed, o, n))
                g = np.zeros(lib().lcmc_mlp_num_params(h), np.float32)
                assert lib().lcmc_mlp_gradients(h, fp(x[:256].copy()), fp(want[:256].copy()), 256, fp(g), None) == 0
                lib().lcmc_mlp_destroy(h)
        except Exception as e:  # (a thread's exception would be lost)
            failed.append((seed, repr(e)))

    threads = [threading.Thread(target=work, args=(s,)) for s in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
