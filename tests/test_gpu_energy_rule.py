"""The total energy by cells or by particles, whichever a system's particles per
cell call for: gases on both sides of the rule, alone and in one batch, NVT and
NPT boxes, against the per-particle sum of the upload.  Both sum the same FP64
terms (1e-12 of the total, as in the cell kernel's own test), and energies taken
between sweeps leave the moves as they are.
"""
import numpy as np
import pytest

import parellel_mc_mpi_for_liquidcrystalsystems_b200 as lcmc

pytestmark = pytest.mark.gpu


def params(n, L, r, npt, precision):
    return lcmc.default_params(mc_ensemble_type=2 if npt else 1, num_particles=n, system_density=n / L**3,
                               system_pressure=0.1, npt_max_dlnV=0.02, gb_kappa=3.0, gb_kappa_prime=5.0, gb_mu_exponent=2.0,
                               gb_nu_exponent=1.0, cutoff_radius=4.0, max_displacement=0.1, max_rotation=0.1,
                               init_lattice=1, precision_mode=precision, rng_seed=r + 1)


SYSTEMS = [(4000, 60.0), (8000, 42.0), (300, 12.0), (1000, 70.0), (12000, 36.0)]  # 1.5, 8, 37 (two cells an edge), 0.2, 24


@pytest.mark.parametrize("npt", [False, True])
@pytest.mark.parametrize("precision", [0, 1])
def test_total_either_way(npt, precision):
    ps = [params(n, L, r, npt, precision) for r, (n, L) in enumerate(SYSTEMS)]
    with lcmc.GBSystem(ps) as batch:
        for r in range(len(ps)):
            batch.get_initial_config(r)
        want = [batch.stats(r)["energy"] for r in range(len(ps))]  # (per particle, once every replica is there)
        for r, p in enumerate(ps):
            assert batch.tot_ene(replica=r) == pytest.approx(want[r], rel=1e-12, abs=1e-12 * p.num_particles)
            with lcmc.GBSystem([p]) as s:
                s.get_initial_config()
                assert s.tot_ene() == pytest.approx(want[r], rel=1e-12, abs=1e-12 * p.num_particles)


def test_energy_between_sweeps_leaves_the_moves():
    p = params(8000, 42.0, 1, False, 1)
    out = []
    for look in (False, True):
        with lcmc.GBSystem([p]) as s:
            s.get_initial_config()
            for _ in range(4):
                s.sweep(1)
                if look:
                    s.tot_ene()
            out.append([np.array(a) for a in s.download()[0]] + [np.array(s.outcomes())])
    for a, b in zip(*out):
        assert np.array_equal(a, b)
