"""GPU: nhw_estimate_dt_noalloc over the sizes and values at which its columns split differently.

One column, chunks of levels that do not divide the height, whole columns
(77,824 columns and more), more columns than one pass of the grid, and values
that decide the minimum in each direction or must be skipped: a vertical
velocity that limits dt in one cell, NaN, infinite velocities, dry (zero) and
negative depths.  The reference value is formed in FP64 on the host in the
order of the routine it replaces, and dt must equal it.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 1), (3, 2, 7), (33, 5, 64), (256, 8, 10), (301, 64, 5), (304, 256, 2), (305, 256, 3), (2050, 1030, 1)]
WHAT = ["plain", "w_limits", "v_limits", "nan", "inf", "dry", "negative_depth"]


def _reference(U, V, W, D, dsig, p):
    c = slice(2, -2)
    u, v, w, d, ds = U[c, c, c], V[c, c, c], W[c, c, c], D[c, c][None], dsig[c][:, None, None]
    small = np.float64(np.float32(1.0e-16))

    def floor(x):     # a > Small ? a : Small
        return np.where(x > small, x, small)
    with np.errstate(all="ignore"):
        s = np.sqrt(np.float64(np.float32(9.81)) * d)
        cand = [p["dx"] / floor(np.abs(u) + s), p["dy"] / floor(np.abs(v) + s), ds * d / floor(np.abs(w))]
    m = 10000000.0
    for a in cand:
        a = np.broadcast_to(a, u.shape)
        a = a[~np.isnan(a)]
        if a.size:
            m = min(m, a.min())
    return min(np.float64(np.float32(1.05)) * p["dt_old"], p["cfl"] * m, 10000000.0, p["dt_max"])


@pytest.mark.parametrize("what", WHAT)
@pytest.mark.parametrize("size", SIZES, ids=lambda s: "x".join(map(str, s)))
def test_dt_equals_the_reference(size, what, gpu_lib):
    torch = pytest.importorskip("torch")
    from nhwave_gb300 import lib
    M, N, K = size
    g = np.random.default_rng(11)
    U, V, W = (0.3 * g.standard_normal((K + 4, N + 4, M + 4)) for _ in range(3))
    D = 1.0 + 0.2 * g.random((N + 4, M + 4))
    dsig = 0.5 / K + g.random(K + 4) / K
    k, j, i = K + 1, N + 1, M + 1      # the last interior cell
    if what == "w_limits":
        W[k, j, i] = -500.0
    elif what == "v_limits":
        V[k, j, i] = -80.0
    elif what == "nan":
        U[2, 2, 2] = V[k, j, i] = W[2, 2, 2] = np.nan
        D[j, i] = np.nan
    elif what == "inf":
        V[k, j, i] = -np.inf
    elif what == "dry":
        D[j, i] = 0.0
    elif what == "negative_depth":
        D[j, i] = -0.25
    U[0], V[:, 0], W[:, :, 0] = 1e9, 1e9, 1e9      # ghosts are not read
    p = dict(dx=0.1, dy=0.12, cfl=0.5, dt_old=1e6, dt_max=1e6)
    arrs = [torch.from_numpy(np.ascontiguousarray(a)).to("cuda") for a in (U, V, W, D, dsig)]
    out = torch.full((1,), -1.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    for _ in range(2):      # the second call finds the first one's scratch
        st = lib.load().nhw_estimate_dt_noalloc(*[a.data_ptr() for a in arrs], M, N, K, p["dx"], p["dy"], p["cfl"],
                                                p["dt_old"], p["dt_max"], out.data_ptr(), None)
        assert st == lib.OK, lib.last_error()
        torch.cuda.synchronize()
        assert float(out.cpu()[0]) == _reference(U, V, W, D, dsig, p)
