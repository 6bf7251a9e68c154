"""A batch whose systems differ in kappa, kappa' or eps0 runs the same FP32 pair
terms (mu = 2, nu = 1, sigma0 = 1) as each system alone: every attempt's energy
change, the FP32 screen's decisions and the energies are the same bits.
"""
import numpy as np
import pytest

import parellel_mc_mpi_for_liquidcrystalsystems_b200 as lcmc

pytestmark = pytest.mark.gpu

SHAPES = [(3.0, 5.0, 1.0), (2.8, 5.0, 1.0), (3.0, 4.0, 1.0), (3.0, 5.0, 1.5)]


def params(r, n, npt):
    kappa, kappa_prime, eps0 = SHAPES[r]
    return lcmc.default_params(mc_ensemble_type=2 if npt else 1, num_particles=n + 100 * r, system_density=0.28,
                               system_pressure=2.0, npt_max_dlnV=0.01, gb_kappa=kappa, gb_kappa_prime=kappa_prime,
                               gb_epsilon0=eps0, gb_mu_exponent=2.0, gb_nu_exponent=1.0, cutoff_radius=4.0,
                               max_displacement=0.1, max_rotation=0.1, init_lattice=1, init_orientation_cone_deg=20.0,
                               precision_mode=1, rng_seed=r + 1)


def run(ps, screen, sweeps):
    with lcmc.GBSystem(ps) as s:
        for r in range(len(ps)):
            s.get_initial_config(r)
        if screen:
            s.set_fp32_screen(True)
        s.record_moves(True)
        rows = [[] for _ in ps]
        for _ in range(sweeps):
            try:
                s.sweep(1)
            except lcmc.LcmcError as e:
                if e.code != lcmc._lib.EDRIFT:
                    raise
                s.clear_error_flags()
            for r in range(len(ps)):
                st = s.stats(r)
                rows[r].append((s.move_records(r)[0], st["energy"], st["volume_accepted"], st["volume_stage1_rejected"]))
        return rows


@pytest.mark.parametrize("n,npt", [(6000, False), (6000, True), (40000, False)])
def test_batch_equals_alone(n, npt):
    ps = [params(r, n, npt) for r in range(len(SHAPES))]
    got = run(ps, npt, 12)
    for r, p in enumerate(ps):
        for (a, *x), (b, *y) in zip(got[r], run([p], npt, 12)[0]):
            assert np.array_equal(a, b) and x == y
