"""FP64 sweeps on a GPU with too little room for the records' scratch: it is made
smaller (more batches, more cells attempted sequentially), and the moves are the
same, bit for bit.
"""
import numpy as np
import pytest
import torch

import parellel_mc_mpi_for_liquidcrystalsystems_b200 as lcmc

pytestmark = pytest.mark.gpu


def system():
    s = lcmc.GBSystem(lcmc.default_params(
        num_particles=100000, system_density=0.30, gb_kappa=3.0, gb_kappa_prime=5.0, gb_mu_exponent=2.0, gb_nu_exponent=1.0,
        cutoff_radius=4.0, max_displacement=0.1, max_rotation=0.1, init_lattice=1, init_orientation_cone_deg=20.0,
        precision_mode=0, rng_seed=5))
    s.get_initial_config()
    return s


def test_scratch_shrinks():
    with system() as s:
        s.sweep(2)
        want, outcomes = [np.array(a) for a in s.download()[0]], np.array(s.outcomes())
    held = []
    with system() as s:
        try:
            for size in (1 << 30, 32 << 20):  # all but 128 to 160 MB of the GPU (the full scratch takes 260)
                while torch.cuda.mem_get_info()[0] - size > 128 << 20:
                    held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
            s.sweep(2)
        finally:
            held.clear()
            torch.cuda.empty_cache()
        got = [np.array(a) for a in s.download()[0]]
        assert np.array_equal(np.array(s.outcomes()), outcomes)
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
