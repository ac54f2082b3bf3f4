"""Q planes and batches of small frames: the FP32 plane path (tensor-core spreading of 32 x 32
tiles, passes X and Z) against the FP64 direct sum at the edges of its tiles, chunks and widths, and
frames run in batches against the same frames one by one, on planes and small volumes."""
import numpy as np
import pytest

import oracle
from helpers import rel_l2
from mp_tools_gb300 import _lib, sql
from mp_tools_gb300.sqom import QGrid, SqomJob

pytestmark = pytest.mark.gpu


def _frames(rng, F, n, box):
    fr = np.zeros((F, n, 4), np.float32)
    fr[..., :3] = rng.uniform(-box / 2, box / 2, (F, n, 3))
    return fr


@pytest.mark.parametrize("eps", [1e-2, 1e-3, 1e-5, 1e-7])
@pytest.mark.parametrize("n,counts,m,centre,window", [
    (1, [1], 10, 0.0, False), (129, [100, 29], 33, 0.0, False), (1000, [400, 400, 200], 150, 0.0, True),
    (2047, [2000, 47], 97, 1.25, False), (4096, [4096], 20, 0.5, True)])
def test_plane_against_direct_sum(cuda, eps, n, counts, m, centre, window):
    """Error bound: the kernel's truncation, a few eps, plus FP32 rounding (the bound 3e-6 is 8x
    the 4e-7 that the volumes' FP32 pipeline shows)."""
    box, F = 20.0, 3
    rng = np.random.default_rng(n + m)
    fr = _frames(rng, F, n, box)
    if n > 2000:
        fr[:, :n // 2, :2] = fr[:, :1, :2]          # half the atoms project onto one point
    grid = QGrid(_lib.BULK, (1, 1, 1), n_bz=(m + 0.25) * 2 * np.pi / box, a_par=(box,) * 3, ndim=2,
                 q_center=(centre, 0.0, 0.0))
    job = SqomJob(grid, species_counts=counts, n_frames=F, eps=eps, window=window)
    try:
        assert job.uses_pruned_fft()
        job.set_frames(fr)
        job.transform()
        cs = job.amplitudes()
    finally:
        job.close()
    for t in range(F):
        r = fr[t, :, :3].astype(np.float64)
        x = [r[:, k] * float(grid.tpe[k]) for k in range(2)]
        c = np.exp(-2j * np.pi * centre * r[:, 0])
        if window:
            c = c * (1 + np.cos(x[0])) * (1 + np.cos(x[1])) * 0.25
        ref = oracle.dirft2d1(x[0], x[1], c, -1, grid.n_q[0], grid.n_q[1])
        assert rel_l2(cs[t], ref) < 5 * eps + 3e-6, (t, eps)


@pytest.mark.parametrize("ndim,F,counts,weight,store", [
    (2, 2, [700, 300], 1, True), (2, 7, [500, 300, 201], 3, False), (2, 40, [999], 1, False),
    (3, 5, [600, 300, 101], 1, True), (3, 33, [512], 3, False)])
def test_batched_frames_equal_single_frames(cuda, ndim, F, counts, weight, store):
    """A multi-frame call (batches, a remainder among them) and one call per frame: the same sums in
    another order of a tile's records, so FP32 rounding apart (2e-6)."""
    box, m, n = 24.0, 30, sum(counts)
    rng = np.random.default_rng(F)
    fr = _frames(rng, F, n, box)
    grid = QGrid(_lib.BULK, (1, 1, 1), n_bz=(m + 0.25) * 2 * np.pi / box, a_par=(box,) * 3, ndim=ndim)
    xff = [[6.4, 3.0, 1.9, 0.7, 1.6, 31.5, 2.0, 85.1, 1.1]] * len(counts)
    job = SqomJob(grid, species_counts=counts, n_frames=F, eps=1e-6, weight_mode=weight,
                  xff=xff, store_species=store)
    try:
        job.set_frames(fr)
        job.transform()
        sq = job.sq_total()
        together = job.amplitudes()
        hist = None if not store or ndim == 2 else job.radial_hist(np.eye(3), [0.26] * 3, 0.1, 3.0, 31)
        for t in range(F):
            job.transform(t, 1)
        alone = job.amplitudes()
        assert rel_l2(together, alone) < 2e-6
        assert rel_l2(sq, job.sq_total()) < 4e-6
        for t in range(F):                              # no frame takes another's place
            assert rel_l2(together[t], alone[t]) < 2e-6
        if hist is not None:
            assert rel_l2(hist, job.radial_hist(np.eye(3), [0.26] * 3, 0.1, 3.0, 31)) < 4e-6
    finally:
        job.close()


@pytest.mark.parametrize("F", [3, 20])
def test_batched_frames_are_reproducible(cuda, F):
    """Under the reproducible order a batch gives the bits of the frames one by one."""
    grid = sql.SqlGrid(4.0, (24.0,) * 3)
    fr = _frames(np.random.default_rng(F), F, 3000, 24.0)
    job = SqomJob(grid, species_counts=[2000, 1000], n_frames=F, eps=1e-6, n_atoms_frame=3000)
    try:
        job.set_option(_lib.OPT_REPRODUCIBLE, 1)
        job.set_frames(fr)
        job.transform()
        together = job.amplitudes()
        for t in range(F):
            job.transform(t, 1)
        assert np.array_equal(together, job.amplitudes())
    finally:
        job.close()
