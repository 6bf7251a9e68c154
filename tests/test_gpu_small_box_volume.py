"""Volume moves of boxes with fewer than four cells along an axis, which the
FP32 kernel and its screen leave to FP64: with the screen switched on such a box
takes the plain test, so its trajectory is that of a run without the screen.
Also a box that shrinks through four cells (64) into three while it runs.
"""
import numpy as np
import pytest

import parellel_mc_mpi_for_liquidcrystalsystems_b200 as lcmc

pytestmark = pytest.mark.gpu

COMMON = dict(mc_ensemble_type=2, system_temperature=0.9, npt_max_dlnV=0.01, gb_kappa=3.0, gb_kappa_prime=5.0,
              gb_mu_exponent=2.0, gb_nu_exponent=1.0, cutoff_radius=4.0, max_displacement=0.1, max_rotation=0.1,
              init_lattice=1, init_orientation_cone_deg=20.0, precision_mode=1)


def run(ps, screen, sweeps):
    with lcmc.GBSystem(ps) as s:
        for r in range(len(ps)):
            s.get_initial_config(r)
        if screen:
            s.set_fp32_screen(True)
        boxes = []
        for _ in range(sweeps):
            try:
                s.sweep(1)
            except lcmc.LcmcError as e:
                if e.code != lcmc._lib.EDRIFT:
                    raise
                s.clear_error_flags()
            boxes.append([s.download(replica=r)[1] for r in range(len(ps))])
        out = [s.download(replica=r)[0] for r in range(len(ps))]
        st = [s.stats(r) for r in range(len(ps))]
    return np.array(boxes), out, st


@pytest.mark.parametrize("grid", [0, 1])
def test_screen_leaves_small_boxes_alone(grid):
    ps = [lcmc.default_params(**dict(COMMON, num_particles=n, system_density=0.30, system_pressure=2.0, cell_grid=grid,
                                     rng_seed=n)) for n in (300, 1000)]
    a, x, sa = run(ps, False, 12)
    b, y, sb = run(ps, True, 12)
    np.testing.assert_array_equal(a, b)
    for u, v in zip(x, y):
        for p, q in zip(u, v):
            np.testing.assert_array_equal(p, q)
    for u, v in zip(sa, sb):
        assert u["accepted"] == v["accepted"] and u["volume_accepted"] == v["volume_accepted"]
        assert u["volume_accepted"] > 0


@pytest.mark.parametrize("screen", [False, True])
def test_box_shrinks_below_four_cells(screen):
    # 16.3 on an edge: four cells of 4.07; a pressure far above the density's takes it below 16
    ps = [lcmc.default_params(**dict(COMMON, num_particles=1250, system_density=1250 / 16.3**3, system_pressure=8.0,
                                     cell_grid=1, rng_seed=3)),
          lcmc.default_params(**dict(COMMON, num_particles=4000, system_density=0.30, system_pressure=2.0, cell_grid=1,
                                     rng_seed=4))]
    boxes, out, st = run(ps, screen, 60)
    edge = boxes[:, 0, 0]
    assert edge[0] > 16.0 and edge[-1] < 16.0
    for r in range(2):
        assert all(np.isfinite(a).all() for a in out[r])
        assert np.isfinite(st[r]["energy"])
