"""FP64 spreading against the FP64 direct sum: planes and volumes at every parity of the width, few and
many points per tile, coinciding points, complex strengths (plan) and packed real pairs (job)."""
import numpy as np
import pytest

import oracle
from helpers import plan_type1, rel_l2
from mp_tools_gb300 import _lib
from mp_tools_gb300.sqom import QGrid, SqomJob

pytestmark = pytest.mark.gpu


def _tol(eps):
    return max(5 * eps, 2e-13)       # the bound the other FP64 parity tests use


@pytest.mark.parametrize("eps", [1e-1, 1e-2, 1e-3, 1e-6, 1e-9, 1e-10, 1e-13, 1e-14])
@pytest.mark.parametrize("dim,modes,n", [(2, (20, 17), 1), (2, (65, 130), 17), (2, (33, 31), 3000),
                                         (3, (12, 9, 20), 15), (3, (22, 33, 17), 2500)])
def test_plan_fp64(cuda, dim, modes, n, eps):
    rng = np.random.default_rng(n + dim)
    x, y, z = rng.uniform(-np.pi, np.pi, (3, n))
    if n > 1000:
        x[: n // 2], y[: n // 2], z[: n // 2] = x[0], y[0], z[0]
    c = rng.normal(size=(2, n)) + 1j * rng.normal(size=(2, n))
    fk = plan_type1(cuda, dim, list(modes), x, y, z, c, -1, eps, _lib.FP64, ntrans=2)
    for t in range(2):
        ref = (oracle.dirft2d1(x, y, c[t], -1, *modes) if dim == 2
               else oracle.dirft3d1(x, y, z, c[t], -1, *modes))
        # (a width-2 or -3 kernel is good to a few eps only on average: the looser bound of 10 eps)
        assert rel_l2(fk[t], ref) < (10 * eps if eps > 1e-4 else _tol(eps)), t


@pytest.mark.parametrize("ndim,counts", [(2, [300, 40, 161]), (3, [300, 41])])
def test_job_pairs_fp64(cuda, ndim, counts):
    box, m, F = 20.0, 26, 2
    n = sum(counts)
    rng = np.random.default_rng(n)
    fr = np.zeros((F, n, 4), np.float32)
    fr[..., :3] = rng.uniform(-box / 2, box / 2, (F, n, 3))
    grid = QGrid(_lib.BULK, (1, 1, 1), n_bz=(m + 0.25) * 2 * np.pi / box, a_par=(box,) * 3, ndim=ndim)
    b = [0.3, -0.7, 1.1][:len(counts)]
    job = SqomJob(grid, species_counts=counts, n_frames=F, precision=_lib.FP64, eps=1e-11,
                  weight_mode=_lib.WEIGHT_NEUTRON, b_coh=b)
    try:
        job.set_frames(fr)
        job.transform()
        cs = job.amplitudes()
    finally:
        job.close()
    w = np.repeat(b, counts).astype(complex)
    for t in range(F):
        x = [fr[t, :, k].astype(np.float64) * float(grid.tpe[k]) for k in range(3)]
        ref = (oracle.dirft2d1(x[0], x[1], w, -1, *grid.n_q[:2]) if ndim == 2
               else oracle.dirft3d1(*x, w, -1, *grid.n_q))
        assert rel_l2(cs[t], ref) < 5e-11
