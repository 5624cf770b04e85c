"""GPU: nhw_estimate_dt_noalloc where its products leave the range of doubles.

The vertical candidates dsig D / |W| are divided only where products do not
show them above the horizontal ones.  Velocities of a run that has blown up,
spacings near the smallest number and level thicknesses of both signs over a
negative depth take those products to infinity, to zero and to the wrong order;
dt must equal the host's value all the same.
"""
import numpy as np
import pytest

from test_zz_no_alloc_shapes import _reference

pytestmark = pytest.mark.gpu


def _case(what, M, N, K):
    g = np.random.default_rng(7)
    U, V, W = (0.3 * g.standard_normal((K + 4, N + 4, M + 4)) for _ in range(3))
    D = 1.0 + 0.2 * g.random((N + 4, M + 4))
    dsig = 0.5 / K + g.random(K + 4) / K
    p = dict(dx=0.1, dy=0.12, cfl=0.5, dt_old=1e6, dt_max=1e6)
    k, j, i = K + 1, N + 1, M + 1
    if what == "blown_up":         # dsig D |U| and dx |W| both overflow; the vertical candidate is the smaller
        D[:] = 5000.0
        U[2, j, i], W[k, j, i], p["dx"], p["dy"] = 3e306, -1.5e308, 100.0, 1e200
    elif what == "tiny_spacing":   # dx times the floor of |W| vanishes, and so does the dry column's candidate
        D[j, i] = 0.0
        W[:, j, i] = 0.0
        p["dx"] = p["dy"] = 1e-310
    elif what == "signs":          # thicknesses of both signs over a negative depth: the largest one decides
        dsig[::2] *= -1.0
        D[j, i] = -1e6
        W[:, j, i] = 0.0
    return U, V, W, D, dsig, p


@pytest.mark.parametrize("what", ["blown_up", "tiny_spacing", "signs"])
@pytest.mark.parametrize("size", [(3, 2, 7), (305, 256, 4)], ids=lambda s: "x".join(map(str, s)))
def test_dt_out_of_range(size, what, gpu_lib):
    torch = pytest.importorskip("torch")
    from nhwave_gb300 import lib
    U, V, W, D, dsig, p = _case(what, *size)
    arrs = [torch.from_numpy(np.ascontiguousarray(a)).to("cuda") for a in (U, V, W, D, dsig)]
    out = torch.full((1,), -1.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    st = lib.load().nhw_estimate_dt_noalloc(*[a.data_ptr() for a in arrs], *size, p["dx"], p["dy"], p["cfl"],
                                            p["dt_old"], p["dt_max"], out.data_ptr(), None)
    assert st == lib.OK, lib.last_error()
    torch.cuda.synchronize()
    assert float(out.cpu()[0]) == _reference(U, V, W, D, dsig, p)
