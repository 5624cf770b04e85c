"""GPU: the cumulative iteration count of a run beyond 2^31 iterations.

The count is a 64-bit number; a checkpoint carries it, so a run resumed with a
count just below 2^31 must go on counting past it, by as many iterations as
the same run takes from its own count.  The grids take the three forms of the
kernel that counts: clusters, pairs and single blocks.
"""
import numpy as np
import pytest

from test_gpu_shapes import _case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("krylov", [0, 1, 2])
@pytest.mark.parametrize("shape", [(24, 12, 5), (157, 153, 13), (300, 230, 10)], ids=lambda s: "x".join(map(str, s)))
def test_counts_past_two_to_the_31(shape, krylov, gpu_lib):
    from nhwave_gb300 import lib
    p, depth, eta = _case(*shape, 1, 1e-8)
    p.krylov_kernel = krylov
    g = lib.Scenario(p, depth, eta)
    assert g.step() == 0
    buf = g.save_state()
    s0 = g.scalars()
    assert g.step() == 0
    taken = g.scalars().total_krylov_iters - s0.total_krylov_iters
    assert taken > 0
    # the count and the number of solves stand side by side among the scalars that open the state
    key = np.array([s0.total_krylov_iters, s0.poisson_solves], dtype=np.int64).tobytes()
    raw = buf[:1024].tobytes()
    assert raw.count(key) == 1
    at = raw.index(key)
    start = 2 ** 31 - 2
    buf[at:at + 8] = np.frombuffer(np.int64(start).tobytes(), dtype=np.uint8)
    g.load_state(buf)
    assert g.scalars().total_krylov_iters == start
    assert g.step() == 0
    assert g.scalars().total_krylov_iters == start + taken
    g.close()
