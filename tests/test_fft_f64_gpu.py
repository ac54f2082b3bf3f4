"""Line transforms, FP64: every fine-grid length up to 1,600 (each radix, plan and line count per CTA) on
each axis against the FP64 direct sum, both transform directions, and jobs against the cuFFT path;
FP32: every length of an axis in volume plans of 2^22 points and more."""
import numpy as np
import pytest

import oracle
from helpers import plan_type1, rel_l2
from mp_tools_gb300 import _lib
from mp_tools_gb300.sqom import QGrid, SqomJob

pytestmark = pytest.mark.gpu


def _smooth(n):
    for p in (2, 3, 5):
        while n % p == 0:
            n //= p
    return n == 1


PLANE = [n for n in range(32, 1601, 32) if _smooth(n)]
VOLUME = [n for n in range(48, 500, 16) if _smooth(n)]


@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("n", PLANE)
def test_plane_lengths(cuda, n, axis):
    """eps 1e-11: the truncation, a few 1e-12, is far above the transform's rounding, and any wrong
    twiddle or position shows at order one; bound 5 eps as in the other FP64 parity tests."""
    rng = np.random.default_rng(n)
    m = [15, 15]
    m[axis] = n // 2 - (n // 32) % 2          # odd and even mode counts
    x, y = rng.uniform(-np.pi, np.pi, (2, 300))
    c = rng.normal(size=(2, 300)) + 1j * rng.normal(size=(2, 300))
    sign = 1 if n % 64 else -1
    fk = plan_type1(cuda, 2, m, x, y, x, c, sign, 1e-11, _lib.FP64, ntrans=2)
    for t in range(2):
        assert rel_l2(fk[t], oracle.dirft2d1(x, y, c[t], sign, *m)) < 5e-11


@pytest.mark.parametrize("n", VOLUME)
def test_volume_lengths(cuda, n):
    rng = np.random.default_rng(n)
    axis = (n // 16) % 3
    m = [9, 14, 11]
    m[axis] = n // 2
    x, y, z = rng.uniform(-np.pi, np.pi, (3, 150))
    c = (rng.normal(size=150) + 1j * rng.normal(size=150))[None]
    sign = 1 if n % 32 else -1
    fk = plan_type1(cuda, 3, m, x, y, z, c, sign, 1e-11, _lib.FP64)
    assert rel_l2(fk[0], oracle.dirft3d1(x, y, z, c[0], sign, *m)) < 5e-11


@pytest.mark.parametrize("ndim,F,m,store,window", [(2, 1, 40, False, False), (2, 9, 33, True, True),
                                                   (3, 1, 30, True, False), (3, 6, 17, False, True),
                                                   (3, 2, 128, False, False)])
def test_jobs_equal_cufft(cuda, ndim, F, m, store, window):
    """The same grids and records through cuFFT and through the line passes (batched frames, grids in
    turns at 128^3 modes): FP64 rounding apart, 1e-12."""
    box, counts = 22.0, [300, 200, 45]
    n = sum(counts)
    rng = np.random.default_rng(m)
    fr = np.zeros((F, n, 4), np.float32)
    fr[..., :3] = rng.uniform(-box / 2, box / 2, (F, n, 3))
    grid = QGrid(_lib.BULK, (1, 1, 1), n_bz=(m + 0.25) * 2 * np.pi / box, a_par=(box,) * 3, ndim=ndim)
    out = []
    for cufft in (False, True):
        job = SqomJob(grid, species_counts=counts, n_frames=F, precision=_lib.FP64, eps=1e-9,
                      store_species=store, window=window, no_pruned_fft=cufft)
        try:
            job.set_frames(fr)
            job.transform()
            out.append((job.amplitudes(), job.sq_total()))
            if F > 1:
                job.transform(F - 1, 1)
                assert rel_l2(job.amplitudes()[-1], out[-1][0][-1]) < 1e-12
        finally:
            job.close()
    assert rel_l2(out[0][0], out[1][0]) < 1e-12
    assert rel_l2(out[0][1], out[1][1]) < 1e-6


@pytest.mark.parametrize("n", [32, 288, 480, 576, 800, 864, 1440])
def test_fp32_plane_lengths(cuda, n):
    """FP32 planes at the lengths only they take, both axes, against the direct sum (5 eps + 3e-6)."""
    rng = np.random.default_rng(n)
    counts = [1500, 700]
    m = n // 2
    box = (30.0, 30.0, 30.0)
    for e1, e2 in (((1, 0, 0), (0, 1, 0)), ((0, 1, 0), (1, 0, 0))):
        grid = QGrid(_lib.BULK, (1, 1, 1), e1=e1, e2=e2, n_bz=(m + 0.25) * 2 * np.pi / 30.0, a_par=box, ndim=2)
        fr = np.zeros((2, 2200, 4), np.float32)
        fr[..., :3] = rng.uniform(-15, 15, (2, 2200, 3))
        job = SqomJob(grid, species_counts=counts, n_frames=2, eps=1e-6)
        try:
            assert job.uses_pruned_fft() and job.info()["fine_grid"][:2] == (n, n)
            job.set_frames(fr)
            job.transform()
            cs = job.amplitudes()
        finally:
            job.close()
        ax = [int(np.argmax(np.abs(grid.axis[k]))) for k in range(2)]
        for t in range(2):
            x, y = [fr[t, :, ax[k]].astype(np.float64) * float(grid.tpe[k]) for k in range(2)]
            ref = oracle.dirft2d1(x, y, np.ones(2200, complex), -1, *grid.n_q[:2])
            assert rel_l2(cs[t], ref) < 8e-6


LONG = [n for n in range(48, 2000, 16) if _smooth(n)]


@pytest.mark.parametrize("n", LONG)
def test_fp32_volume_lengths(cuda, n):
    """eps 1e-6: its truncation with FP32 rounding is below the 2e-5 that FP32 plans are held to; a
    wrong twiddle or position shows at order one.  Odd and even mode counts, lines that do not fill
    a CTA, several transforms, both directions."""
    rng = np.random.default_rng(n)
    axis, m = (n // 16) % 3, [9, 14, 11]
    m[axis] = n // 2 - (n // 16) % 2
    if n > 300:
        m[(axis + 1) % 3] = 57
    fine = np.prod([max(32, 2 * k) for k in m])
    ntrans = int(max(1, -(-(1 << 22) // fine)))
    x, y, z = rng.uniform(-np.pi, np.pi, (3, 60))
    c = rng.normal(size=(ntrans, 60)) + 1j * rng.normal(size=(ntrans, 60))
    sign = 1 if n % 32 else -1
    fk = plan_type1(cuda, 3, m, x, y, z, c, sign, 1e-6, _lib.FP32, ntrans=ntrans)
    for t in {0, ntrans // 2, ntrans - 1}:
        assert rel_l2(fk[t], oracle.dirft3d1(*(np.float32(u).astype(float) for u in (x, y, z)), c[t], sign, *m)) < 2e-5
