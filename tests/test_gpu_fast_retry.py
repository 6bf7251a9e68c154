"""FP32 colour phases whose cells exceed the phase kernel's own capacity: they
run again in FP32 with the largest capacity, and only those beyond the class
(or with terms FP32 cannot carry) in FP64.  Slabs of rods denser than the box
was created for fill their cells; every sweep's outcomes are compared with the
FP64 kernel's on the same state (FP32 pair terms decide differently only at
near-ties: at most one attempt in 10^4)."""
import numpy as np
import pytest

import parellel_mc_mpi_for_liquidcrystalsystems_b200 as lcmc

pytestmark = pytest.mark.gpu


def slab(L, height, a, c):
    """Body-centred sites (a apart in the plane, c along z) in the lower part of a box."""
    m, nz = int(L / a), int(height * L / c)
    s = np.arange(2 * m * m * nz)
    b, q = s & 1, s >> 1
    return [np.ascontiguousarray(v) for v in ((q % m + 0.5 * b) * (L / m), (q // m % m + 0.5 * b) * (L / m),
                                              (q // (m * m) + 0.5 * b) * c)]


@pytest.mark.parametrize("height,a,c,low,high", [
    (0.45, 1.15, 3.05, 41, 48),   # cells above 40: beyond the light kernel, within the class
    (0.45, 1.06, 3.00, 49, 64),   # cells above 48: FP64
    (1.00, 1.42, 3.15, 0, 40),    # an ordinary liquid
])
def test_overfull_cells(height, a, c, low, high):
    L = 36.0
    pos = slab(L, height, a, c)
    n = len(pos[0])
    cells = np.floor(np.array(pos) / (L / 8)).astype(int)
    most = np.bincount(cells[0] + 8 * (cells[1] + 8 * cells[2])).max()
    assert low <= most <= high + 8  # counts of a shifted grid differ by a few
    rng = np.random.default_rng(9)
    ct = 1.0 - rng.random(n) * 0.01
    ph = 2 * np.pi * rng.random(n)
    st = np.sqrt(1 - ct * ct)
    kw = dict(num_particles=n, system_density=n / L ** 3, gb_kappa=3.0, gb_kappa_prime=5.0, gb_mu_exponent=2.0,
              gb_nu_exponent=1.0, cutoff_radius=4.0, max_displacement=0.1, max_rotation=0.1, rng_seed=31)
    diff = 0
    with lcmc.GBSystem(lcmc.default_params(precision_mode=1, **kw)) as f, \
            lcmc.GBSystem(lcmc.default_params(precision_mode=0, **kw)) as d:
        state, box = [*pos, st * np.cos(ph), st * np.sin(ph), ct], np.array([L, L, L])
        for _ in range(4):
            for s in (f, d):
                s.upload(*state, box, energy=0.0)
                s.sweep(1)
            diff += int(np.sum(f.outcomes() != d.outcomes()))
            state, box = d.download()
        got = f.stats()
    assert got["kernel"] == 1
    assert diff <= 4 * n // 10000 + 1
    if low > 48:
        assert got["overcap_cells"] > 0
    if high <= 40:
        assert got["overcap_cells"] == 0
