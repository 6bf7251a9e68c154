"""The cell grid's limit of 2^24 cells, 256 along an axis: the largest grid sweeps
as the FP64 kernel does, with rods in the first and the last cells of every axis
and across the periodic seam, and larger ones are refused at creation, also where
the count of cells passes 2^32.
"""
import numpy as np
import pytest

import parellel_mc_mpi_for_liquidcrystalsystems_b200 as lcmc
from parellel_mc_mpi_for_liquidcrystalsystems_b200 import _lib

pytestmark = pytest.mark.gpu


def params(n, L, precision=1, **kw):
    return lcmc.default_params(**dict(dict(
        num_particles=n, system_density=n / L**3, gb_kappa=3.0, gb_kappa_prime=5.0, gb_mu_exponent=2.0, gb_nu_exponent=1.0,
        cutoff_radius=4.0, max_displacement=0.1, max_rotation=0.1, precision_mode=precision, rng_seed=7), **kw))


def test_largest_grid():
    L, m = 256.5 * 4.1, 8
    rng = np.random.default_rng(3)
    # clumps of rods (1.6 apart) around the corner of the box and half way along each axis
    g = 1.6 * (np.arange(m) - 0.5 * (m - 1))
    clump = np.stack(np.meshgrid(g, g, g), -1).reshape(-1, 3) + 1.37
    pos = np.concatenate([clump + np.array(c) * L for c in
                          ([0, 0, 0], [0.5, 0, 0], [0, 0.5, 0], [0, 0, 0.5], [0.996, 0.5, 0.004])]) % L
    n = len(pos)
    u = rng.normal(size=(3, n)) * 0.1 + np.array([[0.0], [0.0], [1.0]])
    state = [*np.ascontiguousarray(pos.T), *(u / np.linalg.norm(u, axis=0))]
    with lcmc.GBSystem(params(n, L)) as f, lcmc.GBSystem(params(n, L, 0)) as d:
        for _ in range(3):
            got = []
            for s in (f, d):
                s.upload(*state, np.full(3, L), energy=0.0)
                s.sweep(1)
                got.append((s.stats()["stencil_candidates"], s.outcomes()))
            assert got[0][0] == got[1][0] > 0
            assert np.sum(got[0][1] != got[1][1]) <= 1  # (a near-tie)
            state = [np.array(a) for a in d.download()[0]]
        assert f.stats()["kernel"] == 1


@pytest.mark.parametrize("cells,grid", [(257.5, 1), (258.5, 0), (1626.5, 0), (3300.5, 1)])
def test_larger_grids_are_refused(cells, grid):
    with pytest.raises(lcmc.LcmcError) as e:
        lcmc.GBSystem(params(2000, cells * 4.1, cell_grid=grid))
    assert e.value.code == _lib.EINVAL
