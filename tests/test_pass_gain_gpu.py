"""Mean power of FP32 plane amplitudes against FP64 ones, for the fine-grid lengths of the passes: what the
rounding of a pass's constants does to all modes alike has to be taken back."""
import numpy as np
import pytest

from mp_tools_gb300 import _lib
from mp_tools_gb300.sqom import QGrid, SqomJob

pytestmark = pytest.mark.gpu

BOX, N = 20.0, 20000


def _power(length, precision, eps, fr):
    grid = QGrid(_lib.BULK, (1, 1, 1), n_bz=(length // 2 + 0.25) * 2 * np.pi / BOX, a_par=(BOX,) * 3, ndim=2)
    job = SqomJob(grid, species_counts=[N // 2, N // 2], n_frames=1, precision=precision, eps=eps)
    try:
        assert precision == _lib.FP64 or (job.info()["fine_grid"][:2] == (length,) * 2 and job.uses_pruned_fft())
        job.set_frames(fr)
        job.transform()
        cs = job.amplitudes_device()[0].clone()
        cs[(grid.n_q[1] // 2) * grid.n_q[0] + grid.n_q[0] // 2] = 0.0     # (the strong mode at Q = 0 alone is exact)
        return float((cs.real.double() ** 2 + cs.imag.double() ** 2).sum())
    finally:
        job.close()


@pytest.mark.parametrize("length", [128, 160, 192, 256, 288, 320, 384, 480, 512, 576, 640, 768, 800, 864, 960, 1024, 1152, 1280,
                                    1440, 1536, 1600])
def test_mean_power(cuda, length):
    """To one FP32 rounding: the errors of single modes (2e-7) and of the rounded deconvolution factors (7e-8
    per axis and mode in power) average out over thousands of modes."""
    fr = np.zeros((1, N, 4), np.float32)
    fr[..., :3] = np.random.default_rng(length).uniform(-BOX / 2, BOX / 2, (1, N, 3))
    assert abs(_power(length, _lib.FP32, 1e-7, fr) / _power(length, _lib.FP64, 1e-12, fr) - 1.0) < 2.0 ** -24
