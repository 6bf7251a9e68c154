"""FP64 colour phases around the capacities of their records, at a cutoff of 5 and
6: particles with 600 to 1100 in-cutoff terms, stencils of 3000 to 4300 slots (96 to
134 chunks of 32), cells within all of them and cells that are attempted
sequentially.  Accept sequences and energies equal the CPU oracle's bit for bit.
"""
import pytest

import test_gpu_exact_phases as phases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,rho,R,kw", [
    (6000, 0.30, 0.0, dict(cutoff_radius=5.0)),   # 94 in a cell, 79 chunks, 640 terms and more with the cell's own
    (7680, 0.30, 0.0, dict(cutoff_radius=6.0)),   # 101 chunks
    (9920, 0.30, 2.0, dict(cutoff_radius=6.0)),   # 131 chunks: sequential
    (5200, 0.42, 0.0, dict(cutoff_radius=6.0)),   # about a thousand terms
])
def test_capacities_bitwise(n, rho, R, kw):
    phases.test_fp64_phases_bitwise(n, rho, R, kw)
