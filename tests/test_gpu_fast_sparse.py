"""The FP32 phase kernel's shape for gases (two warps per cell) makes the moves of
the classes' own shapes, bit for bit: gases up to the density where another shape
is taken, cells that hold more particles than its arrays (run again by the
hand-over kernel), the general pair terms and volume moves.
"""
import numpy as np
import pytest

import parellel_mc_mpi_for_liquidcrystalsystems_b200 as lcmc
from test_gpu_fast_retry import slab

pytestmark = pytest.mark.gpu


def run(cap, n, L, pos, sweeps, **kw):
    with lcmc.GBSystem(lcmc.default_params(**dict(
            dict(num_particles=n, system_density=n / L**3, gb_kappa=3.0, gb_kappa_prime=5.0, gb_mu_exponent=2.0,
                 gb_nu_exponent=1.0, cutoff_radius=4.0, max_displacement=0.2, max_rotation=0.2, npt_max_dlnV=0.01,
                 system_pressure=0.1, init_lattice=1, precision_mode=1, rng_seed=n, cell_capacity=cap), **kw))) as s:
        s.get_initial_config()
        if pos is not None:
            s.upload(*pos, *s.download()[0][3:], np.full(3, L), energy=0.0)
        s.sweep(sweeps)
        return [np.array(a) for a in s.download()[0]], np.array(s.outcomes()), s.stats()


@pytest.mark.parametrize("n,L,kw", [
    (20000, 87.0, {}),                                              # a thousand cells in a phase, two rods in each
    (60000, 100.0, {}),
    (200000, 119.0, {}),                                            # 0.12: nine
    (60000, 100.0, dict(gb_mu_exponent=1.0, gb_nu_exponent=2.0)),
    (30000, 90.0, dict(mc_ensemble_type=2)),
    (0, 100.0, dict()),                                             # a slab of 41 to 48 rods per cell
])
def test_gas_shape_agrees(n, L, kw):
    pos = None
    if n == 0:
        pos = slab(L, 0.2, 1.15, 3.05)
        n = len(pos[0])
    a, out, st = run(0, n, L, pos, 6, **kw)
    assert st["kernel"] == 1 and (pos is None) == (st["overcap_cells"] == 0)
    b, want, sb = run(48, n, L, pos, 6, **kw)  # the 48-particle class's own shape
    assert np.array_equal(out, want) and st["accepted"] == sb["accepted"] and st["energy"] == sb["energy"]
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


def test_cells_above_the_arrays_run_in_fp32():
    """41 to 48 rods in the cells of a slab, more than the light shape's arrays hold: none is left to FP64, so the
    hand-over kernel ran them in FP32."""
    L = 36.0
    pos = slab(L, 0.45, 1.15, 3.05)
    n = len(pos[0])
    with lcmc.GBSystem(lcmc.default_params(num_particles=n, system_density=n / L**3, gb_kappa=3.0, gb_kappa_prime=5.0,
                                           gb_mu_exponent=2.0, gb_nu_exponent=1.0, cutoff_radius=4.0, max_displacement=0.02,
                                           max_rotation=0.02, precision_mode=1, rng_seed=5)) as s:
        s.upload(*pos, np.zeros(n), np.zeros(n), np.ones(n), np.full(3, L), energy=0.0)
        s.sweep(2)
        st = s.stats()
    cells = np.floor(np.array(pos) / (L / 8)).astype(int)
    assert np.bincount(cells[0] + 8 * (cells[1] + 8 * cells[2])).max() > 40
    assert st["kernel"] == 1 and st["fp64_cells"] == 0 and st["attempted"] == 2 * n
