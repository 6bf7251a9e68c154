"""FP32 colour phases whose blocks meet, one after the other, full cells, nearly
empty ones, cells above the capacity and cells of FP64 systems (which they skip):
what one cell fetched into shared memory must be out of the way of the next.
Every replica of such a batch makes the moves it makes alone, bit for bit.
"""
import numpy as np
import pytest

import parellel_mc_mpi_for_liquidcrystalsystems_b200 as lcmc
from test_gpu_fast_retry import slab

pytestmark = pytest.mark.gpu

L = 84.0  # twenty cells along an edge: a thousand in a phase, more than a grid has blocks


def gas(rng, n):
    """Sites of a simple cubic lattice, a random n of them."""
    m = int(L / 1.7)
    s = rng.choice(m**3, n, replace=False)
    return [np.ascontiguousarray((k + 0.5) * (L / m)) for k in (s % m, s // m % m, s // (m * m))]


def replica(kind, seed):
    rng = np.random.default_rng(seed)
    pos = slab(L, 1.0, 1.5, 3.2) if kind == "full" else slab(L, 0.2, 1.06, 3.0) if kind == "slab" else gas(rng, 6000)
    n = len(pos[0])
    ct = 1.0 - rng.random(n) * 0.02
    ph = 2 * np.pi * rng.random(n)
    st = np.sqrt(1 - ct * ct)
    p = lcmc.default_params(num_particles=n, system_density=n / L**3, gb_kappa=3.0, gb_kappa_prime=5.0, gb_mu_exponent=2.0,
                            gb_nu_exponent=1.0, cutoff_radius=4.0, max_displacement=0.1, max_rotation=0.1, rng_seed=seed,
                            cell_capacity=48, precision_mode=0 if kind == "fp64" else 1)
    return p, [*pos, st * np.cos(ph), st * np.sin(ph), ct], np.array([L, L, L])


def run(rs, sweeps):
    with lcmc.GBSystem([p for p, _, _ in rs]) as s:
        for r, (_, state, box) in enumerate(rs):
            s.upload(*state, box, energy=0.0, replica=r)
        s.sweep(sweeps)
        return [([np.array(a) for a in s.download(r)[0]], np.array(s.outcomes(r)), s.stats(r)) for r in range(len(rs))]


def test_blocks_with_cells_of_every_kind():
    rs = [replica(k, 3 + i) for i, k in enumerate(["full", "gas", "fp64", "full", "slab", "fp64", "gas"])]
    batch = run(rs, 4)
    assert [st["kernel"] for _, _, st in batch] == [1, 1, 0, 1, 1, 0, 1]
    assert batch[4][2]["overcap_cells"] > 0
    for one, (state, outcomes, st) in zip(rs, batch):
        (want, wout, wst), = run([one], 4)
        assert np.array_equal(outcomes, wout) and st["accepted"] == wst["accepted"]
        for a, b in zip(state, want):
            assert np.array_equal(a, b)
