"""GPU: face fluxes of narrow grids, where the face kernels change form.

The FP64 blocks across x end below 33 columns, those across y below 0.6 of
their lanes (19 of 32 columns, 38 of 64) and on a single row: sizes on either
side must give the oracle's fluxes and Omega bit for bit, as every FP64 grid
of 65,536 cells and more does.
"""
import pytest

from test_gpu_fp64_faces import test_faces_bit_exact as _faces_bit_exact

pytestmark = pytest.mark.gpu

GRIDS = [(32, 205, 10), (33, 199, 10), (47, 140, 10), (19, 345, 10), (20, 328, 10), (38, 173, 10), (39, 169, 10), (3300, 1, 20),
         (1639, 2, 20), (3, 1100, 20)]


@pytest.mark.parametrize("hllc", [0, 1])
@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "x".join(map(str, g)))
def test_narrow_faces_bit_exact(grid, hllc, oracle_mod, gpu_lib):
    _faces_bit_exact(grid, hllc, oracle_mod, gpu_lib)
