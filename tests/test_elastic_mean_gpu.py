"""The elastic mean that the time maps subtract: a constant series leaves only the rounding of a pairwise
sum over the frames.  Its value is chosen so that a running FP32 sum loses 2^-17 with almost every frame
once it has passed 128."""
import numpy as np
import pytest

from mp_tools_gb300 import _lib
from mp_tools_gb300.sqom import QGrid, SqomJob, TimeAxis

pytestmark = pytest.mark.gpu

VALUE = 1.0 + 2.0 ** -17 - 2.0 ** -23


@pytest.mark.parametrize("F,n_int", [(7, 3), (90, 41), (250, 101), (511, 255), (1500, 301)])
def test_constant_series(cuda, F, n_int):
    """E=const map, E(Q) cut and I(Q,t) at zero frequency.  A sum of F values in pairs, of groups of up to
    F / 2048 eights in a thread, rounds at most log2(F) + 1 + F / 2048 times per value, the division once."""
    grid = QGrid(_lib.BULK, (1, 1, 1), n_bz=20.25 * 2 * np.pi / 20.0, a_par=(20.0,) * 3, ndim=2)
    job = SqomJob(grid, species_counts=[10], n_frames=F, eps=1e-5)
    ta = TimeAxis(F, 0.01, n_int=n_int, j_sq=0)
    w = np.ones(n_int, np.float32)
    try:
        job.amplitudes_device().fill_(VALUE)
        econst = job.sqw_econst(ta, 1, t_wind=w, normalize=False) * (0.5 / n_int)       # |mean left|^2
        cut = job.sqw_dispersion(ta, np.arange(20), n_freq=1, t_wind=w, normalize=False) * (0.5 / n_int)
        iqt = job.iqt(n_int, 0, normalize=False)
    finally:
        job.close()
    bound = 2.0 ** -24 * (np.ceil(np.log2(F)) + 2 + F / 2048)
    bound_groups = bound + 2.0 ** -24 * (F / 8 / 8)      # 32 columns a CTA: eight parts of F / 8 frames, in eights
    assert np.sqrt(cut.max()) <= bound * 1.001
    assert np.sqrt(econst.max()) <= bound_groups * 1.001 and np.sqrt(iqt.max()) <= bound_groups * 1.001
