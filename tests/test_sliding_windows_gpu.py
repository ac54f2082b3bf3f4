"""Sliding-window maps at the edges of the blocks of eight start frames: E=const maps and E(Q) cuts for
window lengths and start-frame counts around multiples of eight, FP32 and FP64, against the sums in
64 bits; cuts with more frequencies than one block of 1,024."""
import numpy as np
import pytest

from helpers import rel_l2
from mp_tools_gb300 import _lib
from mp_tools_gb300.sqom import QGrid, SqomJob, TimeAxis

pytestmark = pytest.mark.gpu


def _job(cuda, F, m, precision, seed):
    grid = QGrid(_lib.BULK, (1, 1, 1), n_bz=(m + 0.25) * 2 * np.pi / 20.0, a_par=(20.0,) * 3, ndim=2)
    job = SqomJob(grid, species_counts=[50], n_frames=F, precision=precision, eps=1e-5)
    rng = np.random.default_rng(seed)
    x = rng.normal(size=(F, grid.n_modes)) + 1j * rng.normal(size=(F, grid.n_modes))
    cs = job.amplitudes_device()
    cs.copy_(cuda.as_tensor(x).to(cs.dtype))
    return job, cs.cpu().numpy().astype(np.complex128)


def _windows(x, n_int, w, j):
    y = x - x.mean(0)
    i = np.arange(n_int)
    ph = w * np.exp(-2j * np.pi * (j - 1) * (i - n_int // 2) / n_int)
    return np.stack([ph @ y[t:t + n_int] for t in range(len(x) - n_int + 1)])


@pytest.mark.parametrize("precision", [_lib.FP32, _lib.FP64])
@pytest.mark.parametrize("F,n_int", [(4, 4), (9, 1), (9, 8), (16, 9), (17, 9), (40, 7), (75, 41), (200, 129)])
def test_windows(cuda, precision, F, n_int):
    """FP32 sums of up to 129 terms: a few times 2^-24 sqrt(129), bound 3e-6; the maps are stored in
    FP32 (bound 3e-7 in FP64, of which 6e-8 is the rounding of the map)."""
    job, x = _job(cuda, F, 30, precision, F + n_int)
    ta = TimeAxis(F, 0.01, n_int=n_int, j_sq=0)
    assert ta.n_int == n_int
    w = np.random.default_rng(1).uniform(0.2, 1.0, n_int).astype(np.float32)
    tol = 3e-6 if precision == _lib.FP32 else 3e-7
    scale = 1.0 / (0.5 * ta.n_frame * n_int)
    path = np.arange(5, 5 + 30 * 7, 7)
    n_freq = max(1, (n_int + 1) // 2)
    try:
        for j in {1, 2, n_freq}:
            got = job.sqw_econst(ta, j, t_wind=w, normalize=False)
            assert rel_l2(got, (np.abs(_windows(x, n_int, w, j)) ** 2).sum(0) * scale) < tol, j
        cut = job.sqw_dispersion(ta, path, n_freq=n_freq, t_wind=w, normalize=False)
        for f in range(n_freq):
            want = (np.abs(_windows(x[:, path], n_int, w, f + 1)) ** 2).sum(0) * scale
            # (the whole cut's norm: a bin of the mean-free series may vanish, as bin 0 does)
            assert np.linalg.norm(cut[:, f] - want) < tol * np.linalg.norm(cut), f
    finally:
        job.close()


def test_cut_with_many_frequencies(cuda):
    F, n_int = 2203, 2200
    job, x = _job(cuda, F, 2, _lib.FP32, 3)
    w = np.ones(n_int, np.float32)
    ta = TimeAxis(F, 0.01, n_int=n_int, j_sq=0)
    try:
        cut = job.sqw_dispersion(ta, [0, 3], n_freq=n_int, t_wind=w, normalize=False)
        y = (x - x.mean(0))[:, [0, 3]]
        want = sum(np.abs(np.fft.fft(y[t:t + n_int], axis=0)) ** 2 for t in range(F - n_int + 1)).T
        assert rel_l2(cut, want / (0.5 * ta.n_frame * n_int)) < 2e-5   # 2^-24 sqrt(2200) and its walk
    finally:
        job.close()
