"""An NPT box that shrinks from five cells through four (4 x 4.141 = 16.56 on an
edge) into three, where the FP32 kernel and the volume move's cell kernel end:
the FP64 phases and the per-particle energies are launched only when a box may
be there.  Beside it, in a batch, an FP64 system of three cells has both launched
in every sweep: the moves, boxes and energies of the two runs are the same bits.
Also with the autotuner called now and then, which must look at the box as it is.
"""
import numpy as np
import pytest

import parellel_mc_mpi_for_liquidcrystalsystems_b200 as lcmc

pytestmark = pytest.mark.gpu

COMMON = dict(mc_ensemble_type=2, system_temperature=0.9, npt_max_dlnV=0.01, gb_kappa=3.0, gb_kappa_prime=5.0,
              gb_mu_exponent=2.0, gb_nu_exponent=1.0, cutoff_radius=4.0, max_displacement=0.1, max_rotation=0.1,
              init_lattice=1, init_orientation_cone_deg=20.0, cell_grid=1)
EDGE, SWEEPS = 18.7, 200


def box():
    return lcmc.default_params(**dict(COMMON, num_particles=1250, system_density=1250 / EDGE**3, system_pressure=12.0,
                                      precision_mode=1, rng_seed=3))


def beside():
    return lcmc.default_params(**dict(COMMON, num_particles=300, system_density=0.25, system_pressure=1.0,
                                      precision_mode=0, rng_seed=5))


def run(ps, screen, tune=None):
    """Boxes, accepted counts, energies and the outcomes' sum after every sweep of the first system; its last state."""
    rows = []
    with lcmc.GBSystem(ps) as s:
        for r in range(len(ps)):
            s.get_initial_config(r)
        if screen:
            s.set_fp32_screen(True)
        for k in range(SWEEPS):
            if tune and k % 25 == 20:
                assert s.autotune(cache=tune)["from_cache"]
            try:
                s.sweep(1)
            except lcmc.LcmcError as e:
                if e.code != lcmc._lib.EDRIFT:
                    raise
                s.clear_error_flags()
            st = s.stats(0)
            rows.append([*st["box"], st["accepted"], st["volume_accepted"], st["energy"], s.outcomes(0).sum(), st["kernel"]])
        return np.array(rows), [np.array(a) for a in s.download(0)[0]]


@pytest.mark.parametrize("screen,tuned", [(False, False), (True, False), (False, True)])
def test_crossing_equals_a_run_with_all_kernels(tmp_path, screen, tuned):
    cache = None
    if tuned:
        cache = tmp_path / "tune"
        with lcmc.GBSystem([box()]) as s:
            s.get_initial_config(0)
            s.autotune(sweeps=1, cache=cache)
        key = cache.read_text().split("\t")[0]
        cache.write_text(f"{key}\t0\t1\t1.0\n")  # the 48-particle class, energies by cells: what runs without the tuner
    want, state = run([box(), beside()], screen)
    edge = want[:, 0]
    assert edge[0] > 18.5 and edge[-1] < 16.5 and want[0, -1] == 1 and want[-1, -1] == 0
    got, other = run([box()], screen, cache)
    assert np.array_equal(got, want)
    for a, b in zip(state, other):
        assert np.array_equal(a, b)
