"""Uploads between the sweeps of a mixed batch.  The two parities of the state
arrays have a captured graph each, made when first needed; a smaller box that
takes an FP32 system below four cells per axis needs more FP64 scratch than the
graph captured before it knows of.  Whatever the number of sweeps between the
uploads, every replica makes the moves it makes alone, bit for bit.
"""
import numpy as np
import pytest

import parellel_mc_mpi_for_liquidcrystalsystems_b200 as lcmc

pytestmark = pytest.mark.gpu


def lattice(n, L, seed):
    rng = np.random.default_rng(seed)
    m = int(np.ceil(n ** (1 / 3)))
    s = np.sort(rng.choice(m**3, n, replace=False))
    u = rng.normal(size=(3, n))
    return [*((k + 0.5) * (L / m) for k in (s % m, s // m % m, s // (m * m))), *(u / np.linalg.norm(u, axis=0))], np.full(3, L)


def params(n, L, **kw):
    return lcmc.default_params(num_particles=n, system_density=n / L**3, gb_kappa=3.0, gb_kappa_prime=5.0, gb_mu_exponent=2.0,
                               gb_nu_exponent=1.0, cutoff_radius=4.0, max_displacement=0.1, max_rotation=0.1, cell_capacity=48,
                               **kw)


def replicas():
    """An FP64 system, an FP32 one that is shrunk, and a larger FP32 one beside which its few cells change no block shape."""
    return [params(300, 13.0, rng_seed=1, precision_mode=0), params(1000, 25.5, rng_seed=2, precision_mode=1),
            params(3000, 34.0, rng_seed=3, precision_mode=1)]


def follow(s, r, which, first, then):
    """`first` sweeps, the upload, `then` sweeps; after each upload and sweep the state of `which`'s replicas."""
    out = []
    for k, (n, L) in enumerate([(300, 13.0), (1000, 25.5), (3000, 34.0)]):
        if k in which:
            s.upload(*lattice(n, L, k)[0], lattice(n, L, k)[1], energy=0.0, replica=r(k))
    for step in range(first + then):
        if step == first and 1 in which:
            s.upload(*lattice(1000, 16.2, 7)[0], lattice(1000, 16.2, 7)[1], energy=0.0, replica=r(1))
        s.sweep(1)
        for k in which:
            out.append([np.array(a) for a in s.download(r(k))[0]] + [np.array(s.outcomes(r(k)))])
    return out


@pytest.mark.parametrize("first", [1, 2, 3])
def test_shrunk_between_sweeps(first):
    with lcmc.GBSystem(replicas()) as s:
        got = follow(s, lambda k: k, (0, 1, 2), first, 5)
        assert [s.stats(r)["kernel"] for r in range(3)] == [0, 0, 1]
    for k in range(3):
        with lcmc.GBSystem([replicas()[k]]) as s:
            want = follow(s, lambda _: 0, (k,), first, 5)
        for a, b in zip(got[k::3], want):
            for x, y in zip(a, b):
                assert np.array_equal(x, y)
