"""Total energy by cells against the per-particle kernel, where the cell kernel
takes another way: cells with more particles than it stages (384), stencils that
are staged in parts (512), empty cells, more replicas than are enumerated
directly (128).  Both sum the same FP64 terms; a term's two forms differ by at
most 12 r / dist ulp with dist >= 0.3 (below that the cell kernel takes the other's
form), 1e-13 of the term, and the terms here are nearly all repulsive: 1e-12 of
the total.
"""
import numpy as np
import pytest

import parellel_mc_mpi_for_liquidcrystalsystems_b200 as lcmc

pytestmark = pytest.mark.gpu


def params(n, L, **kw):
    return lcmc.default_params(num_particles=n, system_density=n / L**3, gb_kappa=3.0, gb_kappa_prime=5.0,
                               gb_mu_exponent=2.0, gb_nu_exponent=1.0, cutoff_radius=4.0, max_displacement=0.1,
                               max_rotation=0.1, **kw)


def rods(rng, n):
    u = rng.normal(size=(3, n))
    return list(u / np.linalg.norm(u, axis=0))


def clump(rng, n, L, size, spacing):
    """n rods on a jittered lattice in a corner block of the box."""
    m = int(np.ceil(size / spacing))
    assert m**3 >= n
    s = rng.choice(m**3, n, replace=False)
    p = (np.stack([s % m, s // m % m, s // (m * m)]) + 0.5) * spacing + rng.uniform(-0.05, 0.05, size=(3, n))
    return [np.ascontiguousarray(v) for v in np.mod(p, L)]


@pytest.mark.parametrize("n,L,size,spacing", [
    (900, 20.0, 6.0, 0.60),    # cells above 384 particles, most cells empty
    (3000, 20.0, 12.0, 0.80),  # stencils above 512
    (2400, 20.0, 20.0, 1.45),  # the whole box
    (40, 40.0, 40.0, 8.0),     # a gas
])
@pytest.mark.parametrize("R", [0.0, 1.5])
def test_total_by_cells(n, L, size, spacing, R):
    rng = np.random.default_rng(n)
    pos = clump(rng, n, L, size, spacing)
    if R:
        d = np.sqrt(sum((p - 0.5 * L) ** 2 for p in pos))
        keep = d > R + 0.5
        pos = [np.ascontiguousarray(p[keep]) for p in pos]
        n = int(keep.sum())
    u = rods(rng, n)
    with lcmc.GBSystem(params(n, L, colloid_radius=R, colloid_wall_option=1 if R else 0)) as s:
        s.upload(*pos, *u, np.array([L, L, L]))
        by_particle = s.stats()["energy"]
        by_cell = s.tot_ene()
    assert by_cell == pytest.approx(by_particle, rel=1e-12, abs=1e-12 * n)


def test_many_replicas():
    rng = np.random.default_rng(5)
    sizes = [(300 + 7 * r, 18.0 + 0.05 * r) for r in range(140)]
    ps = [params(n, L, rng_seed=r + 1) for r, (n, L) in enumerate(sizes)]
    with lcmc.GBSystem(ps) as s:
        for r, (n, L) in enumerate(sizes):
            s.upload(*clump(rng, n, L, L, L / 11.0), *rods(rng, n), np.array([L, L, L]), replica=r)
        want = [s.stats(r)["energy"] for r in range(140)]  # (computed once every replica has its configuration)
        for r in range(0, 140, 13):
            assert s.tot_ene(replica=r) == pytest.approx(want[r], rel=1e-12, abs=1e-10)
