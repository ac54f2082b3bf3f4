"""Per-species amplitudes of masked species are zero, also
where the job's memory held another job's amplitudes before: |Q| histogram and atom-pair maps, FP32 and
FP64, planes and volumes, and slabs of different heights."""
import numpy as np
import pytest

from mp_tools_gb300 import _lib
from mp_tools_gb300.sqom import QGrid, SqomJob, TimeAxis

pytestmark = pytest.mark.gpu

BOX, F, COUNTS = 20.0, 6, [300, 200, 100]


def _job(grid, mask, precision, **kw):
    return SqomJob(grid, species_counts=COUNTS, n_frames=F, precision=precision, eps=1e-5, mask=mask,
                   store_species=True, stream_ordered=True, **kw)


def _frames():
    fr = np.zeros((F, sum(COUNTS), 4), np.float32)
    fr[..., :3] = np.random.default_rng(8).uniform(-BOX / 2, BOX / 2, (F, sum(COUNTS), 3))
    return fr


def _grid(ndim):
    return QGrid(_lib.BULK, (1, 1, 1), n_bz=16.25 * 2 * np.pi / BOX, a_par=(BOX,) * 3, ndim=ndim)


@pytest.mark.parametrize("precision", [_lib.FP32, _lib.FP64])
@pytest.mark.parametrize("ndim", [2, 3])
@pytest.mark.parametrize("mask", [[1, 0, 1], [0, 1, 0], [0, 0, 0]])
def test_masked_species_have_zero_amplitudes(cuda, precision, ndim, mask):
    grid, fr, ta = _grid(ndim), _frames(), TimeAxis(F, 0.01)
    dq = np.asarray(grid.tpe, np.float64)
    for m in ([1, 1, 1], mask):          # the second job takes the memory that the first gave back
        job = _job(grid, m, precision)
        try:
            job.set_frames(fr)
            job.transform()
            hist = job.radial_hist(np.eye(3), dq, 0.5, 4.0, 9)
            pair = [job.sqw_econst(ta, 1, atom_pair=(s, s)) for s in range(3)]
            cut = [job.sqw_dispersion(ta, np.arange(8), atom_pair=(s, s)) for s in range(3)]
        finally:
            job.close()
        for s in range(3):
            assert (hist[s].any(), hist[:, s].any()) == (bool(m[s]),) * 2, (m, s)
            assert pair[s].any() == bool(m[s]) and cut[s].any() == bool(m[s]), (m, s)


def test_masked_species_on_slabs(cuda):
    """The rows of the store move when the last slab is thinner than the others."""
    grid, fr, ta = _grid(3), _frames(), TimeAxis(F, 0.01)
    nz = grid.n_q[2]
    step = nz // 2 + 1
    job = _job(grid, [1, 0, 1], _lib.FP32, q_slab=step)
    try:
        job.set_frames(fr)
        for z0 in (0, step, 0):
            job.set_q_slab(z0)
            job.transform()
            assert not job.sqw_econst(ta, 1, atom_pair=(1, 1)).any(), z0
            assert job.sqw_econst(ta, 1, atom_pair=(2, 2)).all(), z0
    finally:
        job.close()
