"""The FP32 phase kernel's shape follows the particles of the neighbour cells: in
boxes whose cells are as wide as the count allows (30 and 34 rods to a cell, 800
and 900 neighbours) the larger arrays are taken.  Whatever the shape and the
capacity class, the moves are the same, bit for bit, with no cell left to FP64.
"""
import numpy as np
import pytest

import parellel_mc_mpi_for_liquidcrystalsystems_b200 as lcmc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,rho", [
    (30157, 0.30),   # ten cells along an edge, one block per SM: 30 to a cell
    (49000, 0.31),   # twelve, 216 cells in a phase: 28
    (60500, 0.33),   # twelve, 35
    (20000, 0.30),   # ten, 20: the light shape
])
def test_shapes_agree(n, rho):
    kw = dict(num_particles=n, system_density=rho, gb_kappa=3.0, gb_kappa_prime=5.0, gb_mu_exponent=2.0,
              gb_nu_exponent=1.0, cutoff_radius=4.0, max_displacement=0.1, max_rotation=0.1, init_lattice=1,
              init_orientation_cone_deg=20.0, precision_mode=1, rng_seed=n)
    with lcmc.GBSystem(lcmc.default_params(**kw)) as s:
        s.get_initial_config()
        s.sweep(30)
        state, box = s.download()
        state, box = [np.array(a) for a in state], np.array(box)
    out = []
    for cap in (0, 56, 64):
        with lcmc.GBSystem(lcmc.default_params(cell_capacity=cap, **kw)) as s:
            s.upload(*state, box, energy=0.0)
            s.sweep(2)
            out.append([np.array(a) for a in s.download()[0]])
            st = s.stats()
            assert st["kernel"] == 1 and st["fp64_cells"] == 0
    for other in out[1:]:
        for a, b in zip(out[0], other):
            np.testing.assert_array_equal(a, b)
