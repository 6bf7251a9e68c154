"""FP64 decisions in rounds of three attempts, every pattern of outcomes at once:
cells whose particles end a round with one, two or three attempts, that are
empty, and of every class of own-cell chunks, up to and beyond a cell per SM
(above that a warp per cell takes them one by one).  Accept sequences and
energies equal the CPU oracle's bit for bit.
"""
import pytest

import test_gpu_exact_phases as phases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,rho,R,kw", [
    (200, 0.01, 0.0, {}),                           # mostly empty cells
    (1000, 0.20, 0.0, {}),                          # two chunks
    (8192, 0.30, 3.0, {}),                          # three chunks, colloid
    (1001, 0.30, 0.0, dict(max_displacement=1.0)),  # five chunks, few accepted
    (1250, 0.30, 0.0, dict(max_displacement=0.01, max_rotation=0.01)),  # nine chunks, nearly all accepted
    (33000, 0.30, 0.0, dict(init_lattice=1, init_orientation_cone_deg=20.0)),  # 125 cells in a phase
    (45000, 0.30, 0.0, dict(init_lattice=1, init_orientation_cone_deg=20.0)),  # 216
])
def test_rounds_bitwise(n, rho, R, kw):
    phases.test_fp64_phases_bitwise(n, rho, R, kw)
