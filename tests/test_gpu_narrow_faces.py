"""GPU: narrow grids, where the face kernels and the assembly change form.

The FP64 blocks across x end below 33 columns, those across y below 0.6 of
their lanes (19 of 32 columns, 38 of 64) and on a single row: sizes on either
side must give the oracle's fluxes and Omega bit for bit, as every FP64 grid
of 65,536 cells and more does.  The Poisson assembly takes narrow grids in
narrow blocks: steps must be the oracle's within the bounds of every grid.
"""
import pytest

from test_gpu_fp64_faces import test_faces_bit_exact as _faces_bit_exact
from test_gpu_mg_tiles import _against_oracle
from test_gpu_shapes import _case

pytestmark = pytest.mark.gpu

GRIDS = [(32, 205, 10), (33, 199, 10), (47, 140, 10), (19, 345, 10), (20, 328, 10), (38, 173, 10), (39, 169, 10), (3300, 1, 20),
         (1639, 2, 20), (3, 1100, 20)]


@pytest.mark.parametrize("hllc", [0, 1])
@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "x".join(map(str, g)))
def test_narrow_faces_bit_exact(grid, hllc, oracle_mod, gpu_lib):
    _faces_bit_exact(grid, hllc, oracle_mod, gpu_lib)


# widths at which the assembly's blocks change shape, and one more than a block's columns: 2 x 78, 8 x 30, 30 x 8, 78 x 2
ASSEMBLY = [(1, 79, 3), (2, 78, 2), (3, 40, 3), (9, 31, 3), (16, 61, 4), (33, 30, 3), (61, 9, 2), (79, 2, 3), (157, 1, 3)]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("shape", ASSEMBLY, ids=lambda s: "x".join(map(str, s)))
def test_assembly_of_narrow_grids(shape, precision, oracle_mod, gpu_lib):
    p, depth, eta = _case(*shape, precision, 1e-13 if precision == 0 else 1e-10)
    po, _, _ = _case(*shape, 0, 1e-13)
    _against_oracle(p, po, depth, eta, oracle_mod)
