"""GPU: where the multigrid cycle hands over to its single block.

GMRES forms its basis vector in level 0's first passes, and on its own where
the block has level 0 too.  The block takes the last levels, always the coarsest among them, whatever
mg_cta_columns says: below the coarsest level's 8 to 32 columns every level but
it must run outside the block, and the pressure must be solved as the oracle
does (the bounds that every FP64 and FP32+IR grid is held to).
"""
import pytest

from test_gpu_mg_tiles import _against_oracle
from test_gpu_shapes import _case

pytestmark = pytest.mark.gpu


# a hierarchy of three levels, of one, and with a level above the tiles' size
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("columns", [1, 8, 31])
@pytest.mark.parametrize("shape", [(24, 12, 6), (8, 4, 5), (90, 61, 4)], ids=lambda s: "x".join(map(str, s)))
def test_block_takes_the_coarsest_level(shape, columns, precision, oracle_mod, gpu_lib):
    p, depth, eta = _case(*shape, precision, 1e-13 if precision == 0 else 1e-10)
    po, _, _ = _case(*shape, 0, 1e-13)
    p.mg_cta_columns = columns
    _against_oracle(p, po, depth, eta, oracle_mod)


# levels of 64 columns and fewer are the block's from level 0 on; the others have a level above it
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("shape", [(8, 8, 5), (16, 4, 3), (5, 4, 9), (60, 1, 4), (13, 5, 4), (8, 9, 21)],
                         ids=lambda s: "x".join(map(str, s)))
def test_gmres_on_small_grids(shape, precision, oracle_mod, gpu_lib):
    p, depth, eta = _case(*shape, precision, 1e-13 if precision == 0 else 1e-10)
    po, _, _ = _case(*shape, 0, 1e-13)
    p.krylov_kernel = 2
    _against_oracle(p, po, depth, eta, oracle_mod)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [34, 60, 100, 301])
@pytest.mark.parametrize("along_y", [False, True], ids=["x", "y"])
def test_rows_do_not_depend_on_the_spacing_across(n, along_y, precision, gpu_lib):
    """A row of cells has no coupling across it, so a wider cell must cost its
    solves no more than a few iterations (a fifth, and two for the rounding)."""
    from nhwave_gb300 import lib
    its = []
    for ratio in (1.0, 4.0):
        p, depth, eta = _case(*((1, n) if along_y else (n, 1)), 8, precision, 1e-11 if precision == 0 else 1e-8)
        p.dx, p.dy = (0.1 * ratio, 0.1) if along_y else (0.1, 0.1 * ratio)
        g = lib.Scenario(p, depth, eta)
        g.run(4)
        s = g.scalars()
        its.append(s.total_krylov_iters / s.poisson_solves)
        g.close()
    assert its[1] <= 1.2 * its[0] + 2.0, its


# narrow levels at the limits of the tiles: 320 (FP64) and 512 (FP32) of them, one more, and a row of 4096 columns
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("shape", [(1280, 3, 2), (1281, 3, 2), (2, 2048, 2), (2049, 1, 3), (4096, 1, 2)],
                         ids=lambda s: "x".join(map(str, s)))
def test_narrow_levels_step_like_the_oracle(shape, precision, oracle_mod, gpu_lib):
    p, depth, eta = _case(*shape, precision, 1e-13 if precision == 0 else 1e-10)
    po, _, _ = _case(*shape, 0, 1e-13)
    _against_oracle(p, po, depth, eta, oracle_mod)
