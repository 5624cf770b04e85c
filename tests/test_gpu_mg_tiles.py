"""GPU: grids at the edges of the multigrid cycle's tiled levels.

Levels of up to 4096 columns run each half of a V-cycle as one launch of 4 x 4
column tiles, and the last levels as one block's cycle.  Sides that are no
multiple of the tile, a level of exactly 4096 columns and one just above, one
sigma level, and the heights at which a thread takes a second level (33) or the
block's cycle changes form (21, 41) must solve the pressure as the oracle
does: eta and P within the 1e-10 that every FP64 grid is held to, and FP32+IR
eta within 1e-6.
"""
import numpy as np
import pytest

from conftest import rel_l2
from test_gpu_shapes import _case

pytestmark = pytest.mark.gpu

SHAPES = [(64, 64, 2), (65, 64, 2), (63, 65, 3), (7, 9, 21), (13, 6, 33), (10, 9, 41), (66, 3, 1),
          (32, 32, 20)]


# spacings 4, 1/4, 1.5, 2 and 100 times apart: levels that aggregate along one side alone, to the end of a short side;
# the last with more than 512 columns on a broad second level
SPACINGS = [(48, 20, 4, 0.5, 2.0), (48, 20, 4, 2.0, 0.5), (33, 17, 5, 0.5, 0.75), (3, 40, 3, 0.5, 1.0),
            (40, 6, 3, 0.5, 50.0), (60, 50, 3, 0.5, 0.5)]


def _against_oracle(p, po, depth, eta, oracle_mod):
    from nhwave_gb300 import fields as F, lib
    g = lib.Scenario(p, depth, eta)
    o = oracle_mod.Oracle(po, depth.ravel(), eta.ravel())
    for n in range(2):
        assert g.step() == 0 and o.step() == 0
    assert np.array_equal(g.get(F.MASK), o.get(F.MASK))
    sl = o.shape.interior
    r = rel_l2(g.get(F.ETA)[sl(F.ETA)], o.get(F.ETA)[sl(F.ETA)])
    assert r < (1e-10 if p.precision == 0 else 1e-6), f"eta rel L2 {r:.3e}"
    if p.precision == 0:
        r = rel_l2(g.get(F.P)[sl(F.P)], o.get(F.P)[sl(F.P)])
        assert r < 1e-10, f"P rel L2 {r:.3e}"
    g.close()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("grid", SPACINGS, ids=lambda s: "x".join(map(str, s)))
def test_uneven_spacings_step_like_the_oracle(grid, precision, oracle_mod, gpu_lib):
    M, N, K, dx, dy = grid
    p, depth, eta = _case(M, N, K, precision, 1e-13 if precision == 0 else 1e-10)
    po, _, _ = _case(M, N, K, 0, 1e-13)
    p.dx = po.dx = dx
    p.dy = po.dy = dy
    _against_oracle(p, po, depth, eta, oracle_mod)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_tiled_levels_step_like_the_oracle(shape, precision, oracle_mod, gpu_lib):
    p, depth, eta = _case(*shape, precision, 1e-13 if precision == 0 else 1e-10)
    po, _, _ = _case(*shape, 0, 1e-13)
    _against_oracle(p, po, depth, eta, oracle_mod)


# second levels above the tiles' size, which take the colour-split half-sweeps: odd sides, a last aggregate of one row
# or column, a height that is no multiple of the four levels a thread has, and one above 8192 columns
SPLIT = [(133, 130, 5), (259, 129, 1), (131, 127, 9)]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("shape", SPLIT, ids=lambda s: "x".join(map(str, s)))
def test_split_coarse_levels_step_like_the_oracle(shape, precision, oracle_mod, gpu_lib):
    p, depth, eta = _case(*shape, precision, 1e-13 if precision == 0 else 1e-10)
    po, _, _ = _case(*shape, 0, 1e-13)
    _against_oracle(p, po, depth, eta, oracle_mod)


# levels at the edges of the written-out line solves (10 and 20, chunks of 5 and 2), on tiles and on half-sweeps
HEIGHTS = [(24, 12, 5), (24, 12, 6), (24, 12, 10), (24, 12, 11), (24, 12, 19), (70, 61, 10), (70, 61, 11), (70, 61, 21)]
# 153 blocks of 2048 cells, the last of 977: the sums in pairs of blocks
PAIRED = [(157, 153, 13)]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("shape", HEIGHTS + PAIRED, ids=lambda s: "x".join(map(str, s)))
def test_line_solves_and_paired_sums_step_like_the_oracle(shape, precision, oracle_mod, gpu_lib):
    p, depth, eta = _case(*shape, precision, 1e-13 if precision == 0 else 1e-10)
    po, _, _ = _case(*shape, 0, 1e-13)
    _against_oracle(p, po, depth, eta, oracle_mod)
