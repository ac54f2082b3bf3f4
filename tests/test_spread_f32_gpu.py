"""FP32 volume plans at the edges of their spreading: tiles of up to several chunks of 128 points with complex
strengths, every kernel width, clusters inside a tile, across tile and period edges."""
import numpy as np
import pytest

import oracle
from helpers import plan_type1, rel_l2
from mp_tools_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eps", [1e-2, 1e-3, 1e-4, 1e-5, 1e-6, 1e-7])
@pytest.mark.parametrize("n,spread", [(1, 0.0), (127, 0.05), (128, 0.05), (129, 0.3), (257, 0.01), (600, 0.8),
                                      (900, 3.14)])
@pytest.mark.parametrize("centre", [(0.3, -1.0, 2.0), (3.13, -3.13, 0.0)])
def test_clusters(cuda, eps, n, spread, centre):
    """The kernel's truncation, up to ten times eps in the modes at the edge, plus FP32 rounding (3e-6)."""
    rng = np.random.default_rng(n)
    m, ntrans = (21, 24, 30), 2
    r = (np.array(centre)[:, None] + rng.uniform(-spread, spread, (3, n))).astype(np.float32)
    r = ((r + np.pi) % (2 * np.pi) - np.pi).astype(np.float32)
    c = rng.normal(size=(ntrans, n)) + 1j * rng.normal(size=(ntrans, n))
    fk = plan_type1(cuda, 3, m, *r, c, -1, eps, _lib.FP32, ntrans=ntrans)
    for t in range(ntrans):
        ref = oracle.dirft3d1(*r.astype(np.float64), c[t], -1, *m)
        assert rel_l2(fk[t], ref) < 10 * eps + 3e-6
