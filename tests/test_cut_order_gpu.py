"""E(Q) cuts add a frequency's start frames in their order: every run, and every path point with the same
series, gives the same bits."""
import numpy as np
import pytest

from mp_tools_gb300 import _lib
from mp_tools_gb300.sqom import QGrid, SqomJob, TimeAxis

pytestmark = pytest.mark.gpu

GRID = dict(n_bz=4.25 * 2 * np.pi / 20.0, a_par=(20.0,) * 3, ndim=2)


def _job(cuda, series, precision):
    grid = QGrid(_lib.BULK, (1, 1, 1), **GRID)
    job = SqomJob(grid, species_counts=[10], n_frames=len(series), precision=precision, eps=1e-5)
    cs = job.amplitudes_device()
    cs.copy_(cuda.as_tensor(series)[:, None].expand(-1, grid.n_modes).to(cs.dtype))
    return job


@pytest.mark.parametrize("big", [0, 1, 4, 130, 255])
def test_blocks_are_added_in_order(cuda, big):
    """256 blocks of eight start frames (windows of one frame): one block sums to 1 + 2^-24, just between
    two FP32 values, the others to 2^-54 each, which the FP64 sum keeps only in front of the big one; all
    terms and the mean (zero) are exact."""
    F, small = 2048, 2.0 ** -28
    x = np.zeros(F, np.complex128)
    for b in range(F // 8):
        x[8 * b], x[8 * b + 1] = small * (1 + 1j), -small * (1 + 1j)
    x[8 * big:8 * big + 4] = np.array([0.5, -0.5, 2.0 ** -13, -2.0 ** -13]) * (1 + 1j)
    s = 0.0
    for v in (np.abs(x.real) ** 2 + np.abs(x.imag) ** 2).reshape(-1, 8).sum(1):
        s += float(v)
    job = _job(cuda, x, _lib.FP64)
    ta = TimeAxis(F, 0.01, n_int=1, j_sq=0)
    try:
        cut = job.sqw_dispersion(ta, np.zeros(2048, np.int64), n_freq=1, t_wind=[1.0], normalize=False)
    finally:
        job.close()
    assert (cut == np.float32(s * (1.0 / (0.5 * ta.n_frame)))).all()


@pytest.mark.parametrize("precision", [_lib.FP32, _lib.FP64])
@pytest.mark.parametrize("F,n_int,n_freq", [(40, 7, 4), (300, 3, 2), (200, 101, 51), (75, 41, 41), (9000, 1, 1)])
def test_cuts_repeat_bit_for_bit(cuda, precision, F, n_int, n_freq):
    """Few and many blocks, one and several passes over the frequencies, a frequency with more blocks than
    are held at a time; against the sums in 64 bits (bounds of the sliding-window tests)."""
    rng = np.random.default_rng(F)
    x = rng.normal(size=F) + 1j * rng.normal(size=F)
    job = _job(cuda, x, precision)
    ta = TimeAxis(F, 0.01, n_int=n_int, j_sq=0)
    w = np.linspace(0.5, 1.0, n_int).astype(np.float32)
    try:
        cuts = [job.sqw_dispersion(ta, np.zeros(600, np.int64), n_freq=n_freq, t_wind=w, normalize=False)
                for _ in range(3)]
        y = job.amplitudes()[:, 0].astype(np.complex128)
    finally:
        job.close()
    assert all(np.array_equal(c, cuts[0]) for c in cuts) and (cuts[0] == cuts[0][0]).all()
    y = y - y.mean()
    i = np.arange(n_int)
    e = w * np.exp(-2j * np.pi * np.outer(np.arange(n_freq), i) / n_int)
    want = sum(np.abs(e @ y[t:t + n_int]) ** 2 for t in range(F - n_int + 1)) / (0.5 * ta.n_frame * n_int)
    tol = 3e-6 if precision == _lib.FP32 else 3e-7
    assert np.linalg.norm(cuts[0][0] - want) < tol * np.linalg.norm(want)
