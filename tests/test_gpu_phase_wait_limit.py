"""The phase kernels' bounded waits made to run out: with a limit of one try a
block gives up on its first cell's copies, sets the flag, lets the copies land
and leaves; the sweep reports LCMC_ETIMEOUT, nothing faults or hangs, and with
the default limit back a system sweeps as it did before.
"""
import numpy as np
import pytest

import parellel_mc_mpi_for_liquidcrystalsystems_b200 as lcmc
from parellel_mc_mpi_for_liquidcrystalsystems_b200 import _lib
from test_gpu_fast_retry import slab

pytestmark = pytest.mark.gpu

TIMEOUT = 64  # LCMC_F_TIMEOUT


def system(n, rho, precision, pos=None, L=None):
    """A system on a lattice, or on given sites."""
    s = lcmc.GBSystem(lcmc.default_params(
        num_particles=n, system_density=rho, gb_kappa=3.0, gb_kappa_prime=5.0, gb_mu_exponent=2.0, gb_nu_exponent=1.0,
        cutoff_radius=4.0, max_displacement=0.1, max_rotation=0.1, init_lattice=1, init_orientation_cone_deg=20.0,
        precision_mode=precision, rng_seed=n))
    if pos is None:
        s.get_initial_config()
    else:
        s.upload(*pos, np.zeros(n), np.zeros(n), np.ones(n), np.full(3, L), energy=0.0)
    return s


def slab_system():
    """Cells of 41 to 48 particles: above the light block shape's arrays, run again by the hand-over kernel."""
    pos = slab(36.0, 0.45, 1.15, 3.05)
    return system(len(pos[0]), len(pos[0]) / 36.0**3, 1, pos, 36.0)


SYSTEMS = {
    "fp32": lambda: system(60000, 0.30, 1),        # several cells per block
    "fp32_wide": lambda: system(8000, 0.30, 1),    # a block of 512 threads per cell
    "fp32_retry": slab_system,
    "fp64": lambda: system(2000, 0.30, 0),         # records of a cell's attempts copied a round ahead
    "fp64_cells": lambda: system(30000, 0.30, 0),  # a block per cell, a hundred cells
}


def swept(make, sweeps):
    with make() as s:
        s.sweep(sweeps)
        return [np.array(a) for a in s.download()[0]], s.stats()["accepted"]


@pytest.mark.parametrize("name", SYSTEMS)
def test_wait_gives_up_cleanly(name):
    make = SYSTEMS[name]
    want = swept(make, 2)
    try:
        assert _lib.lib().lcmc_set_wait_limit(1) == 0
        with make() as s:
            for _ in range(2):
                with pytest.raises(lcmc.LcmcError) as e:
                    s.sweep(1)
                assert e.value.code == _lib.ETIMEOUT and s.stats()["error_flags"] & TIMEOUT
                s.clear_error_flags()
            state, box = s.download()
            assert all(np.isfinite(a).all() for a in state) and s.stats()["accepted"] < want[1]
    finally:
        _lib.lib().lcmc_set_wait_limit(0)
    got = swept(make, 2)
    assert got[1] == want[1]
    for a, b in zip(got[0], want[0]):
        assert np.array_equal(a, b)
