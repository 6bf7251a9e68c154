"""The hand-over kernel's blocks take cells from a counter: with more cells
than blocks and with fewer, retries among them and stencils larger and smaller than it stages, the
moves repeat bit for bit and are the FP64 kernel's (FP32 pair terms decide
differently only at near-ties: at most one attempt in 10^4).
"""
import numpy as np
import pytest

import parellel_mc_mpi_for_liquidcrystalsystems_b200 as lcmc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,rho,d,least,kw", [
    (100000, 0.28, 1.0, 3 * 8 * 148, {}),  # 900 in a stencil, some of them run again; more than a cell per block
    (60000, 0.30, 0.1, 3 * 8 * 148, dict(init_orientation_cone_deg=180.0, init_lattice=0)),  # overlaps everywhere
    (40000, 0.33, 0.3, 3 * 1000, dict(cell_capacity=20, cutoff_radius=4.6)),  # every cell above the class; 1000 in a stencil
])
def test_many_handed_over(n, rho, d, least, kw):
    p = dict(dict(num_particles=n, system_density=rho, gb_kappa=3.0, gb_kappa_prime=5.0, gb_mu_exponent=2.0,
                  gb_nu_exponent=1.0, cutoff_radius=4.0, max_displacement=d, max_rotation=0.2, init_lattice=1,
                  init_orientation_cone_deg=20.0, rng_seed=n), **kw)
    runs, differ, cells = [], 0, 0
    with lcmc.GBSystem(lcmc.default_params(precision_mode=1, **p)) as f, \
            lcmc.GBSystem(lcmc.default_params(precision_mode=1, **p)) as g, \
            lcmc.GBSystem(lcmc.default_params(precision_mode=0, **p)) as e:
        f.get_initial_config()
        state, box = [np.array(a) for a in f.download()[0]], np.array(f.download()[1])
        for _ in range(3):
            runs = []
            for s in (f, g, e):
                s.upload(*state, box, energy=0.0)
                try:
                    s.sweep(1)
                except lcmc.LcmcError as x:
                    if x.code != lcmc._lib.EDRIFT:
                        raise
                    s.clear_error_flags()
                runs.append(([np.array(a) for a in s.download()[0]], np.array(s.outcomes())))
            assert np.array_equal(runs[0][1], runs[1][1])
            for a, b in zip(runs[0][0], runs[1][0]):
                assert np.array_equal(a, b)
            differ += int(np.sum(runs[0][1] != runs[2][1]))
            state = runs[2][0]
        cells = f.stats()["fp64_cells"]
    assert cells >= least and differ <= 3 * n // 10000
