"""GPU: aggregates that keep coarse levels off the tiles.

mg_aggregate 3 and 8 leave levels whose aggregates do not fill the tiles: they
run half-sweeps, on the colour-split operator or in the natural layout by the
form and the level's size.  Steps must be the oracle's within the bounds of
every grid.
"""
import pytest

from test_gpu_mg_tiles import _against_oracle
from test_gpu_shapes import _case

pytestmark = pytest.mark.gpu


# a coarse level of 600 columns, one of 4160 (aggregates of 3), odd last aggregates
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("aggregate", [3, 8])
@pytest.mark.parametrize("shape", [(90, 60, 6), (240, 156, 2), (61, 47, 5)], ids=lambda s: "x".join(map(str, s)))
def test_aggregates_off_the_tiles(shape, aggregate, precision, oracle_mod, gpu_lib):
    p, depth, eta = _case(*shape, precision, 1e-13 if precision == 0 else 1e-10)
    po, _, _ = _case(*shape, 0, 1e-13)
    p.mg_aggregate = aggregate
    _against_oracle(p, po, depth, eta, oracle_mod)
