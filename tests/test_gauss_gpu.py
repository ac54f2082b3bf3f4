"""FP32 Gaussian-window spectra at 64 to 1,024 frames: every count of frequencies around the half, blocks of
16 modes with remainders."""
import numpy as np
import pytest

from helpers import rel_l2
from mp_tools_gb300 import _lib
from mp_tools_gb300.sqom import QGrid, SqomJob
from oracle.sqom_ref import gauss_spectrum, gauss_window

pytestmark = pytest.mark.gpu

BOX = 20.0


@pytest.mark.parametrize("F", [64, 128, 256, 512, 1024])
@pytest.mark.parametrize("m", [1, 7, 8, 12])
def test_gauss_all_frequencies(cuda, F, m):
    """All F frequencies and the counts around the half, rows of (2 m + 1)^2 modes (ragged blocks of
    16).  FP32 transforms of ten levels: 1e-6; bound 5e-6 of the spectrum (2x for the square)."""
    grid = QGrid(_lib.BULK, (1, 1, 1), n_bz=(m + 0.25) * 2 * np.pi / BOX, a_par=(BOX,) * 3, ndim=2)
    job = SqomJob(grid, species_counts=[50], n_frames=F, eps=1e-5)
    try:
        rng = np.random.default_rng(F + m)
        x = rng.normal(size=(F, grid.n_modes)) + 1j * rng.normal(size=(F, grid.n_modes)) + 3.0
        cs = job.amplitudes_device()
        cs.copy_(cuda.as_tensor(x).to(cs.dtype))
        x = cs.cpu().numpy().astype(np.complex128)
        for n_freq in (1, F // 2, F // 2 + 1, F // 2 + 2, F):
            got = job.sqw_gauss(fwhm_frames=F / 4, n_freq=n_freq, normalize=False)
            want = gauss_spectrum(x, F / 4, n_freq, None, 1.0 / gauss_window(F, F / 4).sum())
            assert rel_l2(got, want) < 5e-6, n_freq
    finally:
        job.close()
