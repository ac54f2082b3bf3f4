"""Crowded tiles in the reproducible order (and without it): up to 1,000 records that coincide to a
thousandth of the box, of one or both species of a packed pair, against the FP64 direct sum.  The bound is
that of the same tiles in the default order: a few eps of truncation plus FP32 rounding (3e-6), which a
sum that loses bits with every further record does not meet."""
import numpy as np
import pytest

import oracle
from helpers import rel_l2
from mp_tools_gb300 import _lib
from mp_tools_gb300.sqom import QGrid, SqomJob

pytestmark = pytest.mark.gpu

BOX = 20.0


@pytest.mark.parametrize("repro", [0, 1])
@pytest.mark.parametrize("eps", [1e-5, 1e-6, 1e-7])
@pytest.mark.parametrize("counts", [[225, 0], [1, 224], [1000], [300, 700]])
def test_coinciding_records(cuda, counts, eps, repro):
    n = sum(counts)
    rng = np.random.default_rng(n)
    fr = np.zeros((1, n, 4), np.float32)
    fr[0, :, :3] = 3.1 + rng.uniform(-0.01, 0.01, (n, 3))
    grid = QGrid(_lib.BULK, (1, 1, 1), n_bz=30.25 * 2 * np.pi / BOX, a_par=(BOX,) * 3, ndim=3)
    job = SqomJob(grid, species_counts=counts, n_frames=1, eps=eps)
    try:
        job.set_option(_lib.OPT_REPRODUCIBLE, repro)
        job.set_frames(fr)
        job.transform()
        cs = job.amplitudes()[0]
    finally:
        job.close()
    m = np.array(grid.n_q)
    pick = rng.integers(0, m, (2000, 3))
    x = [fr[0, :, k].astype(np.float64) * float(grid.tpe[k]) for k in range(3)]
    ref = oracle.dirft_modes(x[0], x[1], x[2], np.ones(n), -1, pick - m // 2)
    assert rel_l2(cs[(pick[:, 2] * m[1] + pick[:, 1]) * m[0] + pick[:, 0]], ref) < 5 * eps + 3e-6
