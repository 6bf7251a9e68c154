"""FP64 colour phases at the edges of their two kernels, bit for bit against the
CPU oracle's canonical sweep: cells above the per-cell capacity and many
in-cutoff terms (dense overlapping boxes, attempted sequentially), one or two
cells per axis (own cell not at slot 13), own-cell slots that straddle chunks of
32, a gas, and a system whose records need more than one batch per phase."""
import numpy as np
import pytest

import oracle_ctypes as oc
import parellel_mc_mpi_for_liquidcrystalsystems_b200 as lcmc

pytestmark = pytest.mark.gpu

COMMON = dict(gb_kappa=3.0, gb_kappa_prime=5.0, gb_mu_exponent=2.0, gb_nu_exponent=1.0, cutoff_radius=4.0,
              max_displacement=0.1, max_rotation=0.1)


@pytest.mark.parametrize("n,rho,R,kw", [
    (160, 0.30, 0.0, {}),                              # one cell
    (620, 0.08, 0.0, {}),                              # gas
    (1300, 0.30, 2.0, {}),                             # 2 cells per axis, ~160 rods each, colloid
    (2200, 0.55, 0.0, {}),                             # ~275 rods per cell: above the cell capacity
    (1500, 0.40, 0.0, {}),                             # many in-cutoff terms per rod
    (4301, 0.33, 0.0, {}),                             # 4 cells per axis
    (2003, 0.30, 0.0, dict(max_displacement=0.5)),     # moves that leave their cell
    (300000, 0.30, 0.0, dict(init_lattice=1, init_orientation_cone_deg=20.0)),  # two batches of records
])
def test_fp64_phases_bitwise(n, rho, R, kw):
    d = dict(COMMON, num_particles=n, system_density=rho, rng_seed=n, precision_mode=0, colloid_radius=R,
             colloid_wall_option=1 if R else 0)
    d.update(kw)
    lp, op = lcmc.default_params(**d), oc.params(**{k: v for k, v in d.items() if k != "init_lattice"})
    a, box = lcmc.lattice(lp)
    state, box = [np.ascontiguousarray(x) for x in a], np.ascontiguousarray(box)
    sweeps = 1 if n > 100000 else 2
    with lcmc.GBSystem(lp) as s:
        s.set_kernel(0)
        s.upload(*state, box, energy=0.0)
        s.sweep(sweeps)
        got, _ = s.download()
        st = s.stats()
    c, k = oc.consts(op, oc.ARITH_CANONICAL), oc.key(op.rng_seed)
    acc = hard = 0
    for sw in range(sweeps):
        if n > 100000:
            o = oc.sweep_parallel(c, k, sw, state, box)
        else:
            o, _, _ = oc.sweep(c, k, sw, state, box)
        acc, hard = acc + o.accepted, hard + o.hardcore_rejected
    for x, y in zip(got, state):
        assert np.array_equal(np.asarray(x).view(np.uint64), y.view(np.uint64))
    assert st["accepted"] == acc and st["hardcore_rejected"] == hard
