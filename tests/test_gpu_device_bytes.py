"""GPU: the device memory that the multigrid hierarchy holds (nhw_device_bytes).

The preconditioner's own arrays are what a scenario holds more than one
preconditioned by lines.  Level 0 has its colour-split operator; a coarse level
its operator, line factors, x and b, the colour-split copy where it is too
large for the tiles, and the tiles' copy of x where it takes them.  Vectors
that only the tiles read are not held for other levels.
"""
import pytest

pytestmark = pytest.mark.gpu

# grid, levels below level 0, those with a colour-split copy, those on tiles (0: level 0 itself)
GRIDS = [((130, 130, 8), [(65, 65), (33, 33), (17, 17), (5, 5)], {1}, {2, 3}),
         ((40, 30, 5), [(20, 15), (5, 4)], set(), {0, 1})]


def _r(n):
    return (n + 255) // 256 * 256


@pytest.mark.parametrize("precision,size", [(0, 8), (1, 4)])
@pytest.mark.parametrize("grid,levels,split,tiles", GRIDS, ids=["split", "tiled"])
def test_multigrid_bytes(grid, levels, split, tiles, precision, size, gpu_lib):
    from nhwave_gb300 import default_params, lib
    M, N, K = grid

    def held(precond):
        p = default_params(Mglob=M, Nglob=N, Kglob=K, dx=0.5, dy=0.5)
        p.precision, p.precond = precision, precond
        return lib.device_bytes(p)

    def colours(m, n):
        return _r(size * 7 * 2 * K * n * ((m + 1) // 2))
    want = colours(M, N) + _r(8 * 2 * 4 * 1024)      # and the partial sums of the persistent solve
    if 0 in tiles:
        want += 2 * _r(size * M * N * K)
    for l, (m, n) in enumerate(levels, 1):
        want += _r(size * 7 * m * n * K) + 4 * _r(size * m * n * K)
        want += colours(m, n) if l in split else 0
        want += _r(size * m * n * K) if l in tiles else 0
    assert held(0) - held(1) == want
