"""Cells without particles are passed by in the colour phases; their results are
written by the rebin.  Gases from one rod in a box to runs of more than 32 empty
cells between two with rods, through the FP32 and the FP64 kernels: the stencil
candidates (whole numbers, summed over every cell) are equal in every sweep, as are
the outcomes but for near-ties of the FP32 terms (none is expected in 10^4
attempts; one is allowed), and the running energy stays that of a recompute,
also where an NPT box's volume moves write the cells' sums between the sweeps.
"""
import numpy as np
import pytest

import parellel_mc_mpi_for_liquidcrystalsystems_b200 as lcmc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,L,npt,grid", [
    (1, 40.0, False, 0), (2, 70.0, False, 1), (40, 70.0, False, 0), (700, 70.0, True, 0), (900, 128.0, False, 1),
    (3000, 60.0, True, 1), (50000, 290.0, False, 0)])
def test_gas(n, L, npt, grid):
    kw = dict(mc_ensemble_type=2 if npt else 1, num_particles=n, system_density=n / L**3, system_pressure=0.02,
              npt_max_dlnV=0.02, gb_kappa=3.0, gb_kappa_prime=5.0, gb_mu_exponent=2.0, gb_nu_exponent=1.0,
              cutoff_radius=4.0, max_displacement=0.4, max_rotation=0.2, init_lattice=1, cell_grid=grid, rng_seed=n)
    with lcmc.GBSystem(lcmc.default_params(precision_mode=1, **kw)) as f, \
            lcmc.GBSystem(lcmc.default_params(precision_mode=0, **kw)) as d:
        f.get_initial_config()
        state, box = [np.array(a) for a in f.download()[0]], np.full(3, L)
        differ, last = 0, [0, 0]
        for _ in range(6):
            got = []
            for k, s in enumerate((f, d)):
                s.upload(*state, box)  # (volume moves of the two may differ)
                s.sweep(1)
                st = s.stats()
                got.append((st["stencil_candidates"] - last[k], s.outcomes()))
                last[k] = st["stencil_candidates"]
                assert st["energy"] == pytest.approx(s.tot_ene(), abs=2e-4 * n)
            assert got[0][0] == got[1][0]
            differ += int(np.sum(got[0][1] != got[1][1]))
            state, box = [np.array(a) for a in d.download()[0]], np.array(d.download()[1])
        assert f.stats()["kernel"] == 1 and differ <= max(1, 6 * n // 10000)
