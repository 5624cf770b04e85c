"""GPU: the FP64 face kernels that share quotients and slopes in blocks.

Grids of 65,536 cells and more take them: rows of 254 faces and one more, 14
and 15 faces across, columns that are no multiple of 32, levels that do not
divide into the chunks, dry land and a front inside a block, HLL and HLLC.
Fluxes and Omega's face values must equal the oracle's bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [(253, 14, 19), (254, 27, 10), (509, 13, 10), (33, 200, 10), (300, 221, 1), (31, 45, 64)]


@pytest.mark.parametrize("hllc", [0, 1])
@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "x".join(map(str, g)))
def test_faces_bit_exact(grid, hllc, oracle_mod, gpu_lib):
    from nhwave_gb300 import default_params, fields as F, lib
    M, N, K = grid
    assert M * N * K >= 65536
    p = default_params(Mglob=M, Nglob=N, Kglob=K, dx=0.7, dy=0.9, dt_ini=0.01, non_hydro=0, hllc=hllc)
    x, y = np.arange(M)[None, :], np.arange(N)[:, None]
    # a basin with dry land in a corner and an island
    depth = 1.5 - 2.0 * np.exp(-((x - 0.9 * M) / (0.2 * M)) ** 2 - ((y - 0.8 * N) / (0.4 * N)) ** 2)
    depth = depth - 3.0 * np.exp(-((x - 0.3 * M) / 9.0) ** 2 - ((y - 0.4 * N) / 5.0) ** 2)
    eta = 0.1 * np.sin(0.13 * x + 0.21 * y)
    uvw = 0.2 * np.random.default_rng(4).standard_normal((3, K, N, M))
    g = lib.Scenario(p, depth.ravel(), eta.ravel(), uvw.ravel())
    o = oracle_mod.Oracle(p, depth.ravel(), eta.ravel(), uvw.ravel())
    sl = o.shape.interior
    for h in (g, o):
        assert h.estimate_dt() == 0
        h.update_mask()
        h.update_vars()
    assert (o.get(F.MASK) == 0).any()
    for s in (1, 2):
        for h in (g, o):
            h.source_terms()
            h.fluxes()
        for n in ("EX", "FX", "GX", "HX", "EY", "FY", "GY", "HY", "FZ", "GZ", "HZ"):
            f = getattr(F, n)
            a, b = g.get(f)[sl(f)], o.get(f)[sl(f)]
            assert np.array_equal(a, b), f"{n} stage {s}: max |d| {np.abs(a - b).max():.3e}"
        for h in (g, o):
            h.eval_duvw(s)
        for n in ("OMEGA", "ETAXL", "ETAXR", "ETAYL", "ETAYR", "U", "W"):
            f = getattr(F, n)
            a, b = g.get(f)[sl(f)], o.get(f)[sl(f)]
            assert np.array_equal(a, b), f"{n} stage {s}: max |d| {np.abs(a - b).max():.3e}"
    g.close()


# FP32+IR, which takes the blocks across y from 2^20 cells on: 14 faces a block and a remainder, columns that are no
# multiple of 32, levels that do not divide into the chunks.  A flux is some twenty roundings of 2^-24 of terms no larger
# than the field's largest, limited slopes included (1.2e-6); Omega's face values are two limited slopes.
FP32_GRIDS = [(1090, 55, 18), (33, 2000, 16)]


@pytest.mark.parametrize("hllc", [0, 1])
@pytest.mark.parametrize("grid", FP32_GRIDS, ids=lambda g: "x".join(map(str, g)))
def test_fp32_y_faces(grid, hllc, oracle_mod, gpu_lib):
    from nhwave_gb300 import default_params, fields as F, lib
    M, N, K = grid
    assert M * N * K >= 1 << 20
    x, y = np.arange(M)[None, :], np.arange(N)[:, None]
    depth = 1.5 + 0.3 * np.sin(0.03 * x) * np.cos(0.05 * y)
    eta = 0.1 * np.sin(0.13 * x + 0.21 * y)
    uvw = (0.2 * np.random.default_rng(4).standard_normal((3, K, N, M))).astype(np.float32).astype(np.float64)
    hs = []
    for prec, make in ((1, lib.Scenario), (0, oracle_mod.Oracle)):
        p = default_params(Mglob=M, Nglob=N, Kglob=K, dx=0.7, dy=0.9, dt_ini=0.01, non_hydro=0, hllc=hllc)
        p.precision = prec
        hs.append(make(p, depth.ravel(), eta.ravel(), uvw.ravel()))
    g, o = hs
    sl = o.shape.interior
    for h in hs:
        assert h.estimate_dt() == 0
        h.update_mask()
        h.update_vars()
        h.source_terms()
        h.fluxes()
    for n in ("EY", "FY", "GY", "HY"):
        f = getattr(F, n)
        a, b = g.get(f)[sl(f)], o.get(f)[sl(f)]
        assert np.abs(a - b).max() <= 1e-5 * np.abs(b).max(), n
    for h in hs:
        h.eval_duvw(1)
    for n in ("OMEGA", "ETAYL", "ETAYR", "V"):
        f = getattr(F, n)
        a, b = g.get(f)[sl(f)], o.get(f)[sl(f)]
        assert np.abs(a - b).max() <= 1e-5 * np.abs(b).max(), n
    g.close()
