"""FP32 volumes at the edges of their kernels: tiles of 0, 1, 16, 17, 224, 225 and more records
(the spreading takes them in chunks of 224 and steps of 16) of one or both species of a packed
pair, at every kernel width; form factors on a Q grid off the origin; all species masked."""
import numpy as np
import pytest

import oracle
from helpers import rel_l2
from mp_tools_gb300 import _lib
from mp_tools_gb300.sqom import QGrid, SqomJob

pytestmark = pytest.mark.gpu

BOX = 20.0
XFF = [[6.4, 3.0, 1.9, 0.7, 1.6, 31.5, 2.0, 85.1, 1.1], [2.3, 20.8, 1.7, 10.2, 0.9, 0.6, 0.4, 51.6, 0.2],
       [12.0, 4.0, 3.1, 0.3, 1.0, 60.0, 0.5, 9.0, 0.7]]


@pytest.mark.parametrize("eps", [1e-2, 1e-3, 1e-4, 1e-5, 1e-6, 1e-7])
@pytest.mark.parametrize("counts", [[1], [0, 1], [16, 1], [17], [200, 24], [1, 224], [225, 0], [300, 700]])
@pytest.mark.parametrize("window", [False, True])
def test_crowded_tiles_against_direct_sum(cuda, eps, counts, window):
    """Frame 0: all points within a thousandth of the box; frame 1: within two tiles' edges.  Error
    bound: the kernel's truncation, a few eps, plus FP32 rounding (3e-6, as for planes)."""
    n, F = sum(counts), 2
    rng = np.random.default_rng(n)
    fr = np.zeros((F, n, 4), np.float32)
    fr[0, :, :3] = 3.1 + rng.uniform(-0.01, 0.01, (n, 3))
    fr[1, :, :3] = -1.7 + rng.uniform(-1.5, 1.5, (n, 3))
    grid = QGrid(_lib.BULK, (1, 1, 1), n_bz=30.25 * 2 * np.pi / BOX, a_par=(BOX,) * 3, ndim=3)
    job = SqomJob(grid, species_counts=counts, n_frames=F, eps=eps, window=window, store_species=True)
    try:
        assert job.uses_pruned_fft()
        job.set_frames(fr)
        job.transform()
        cs = job.amplitudes()
    finally:
        job.close()
    m = np.array(grid.n_q)
    pick = rng.integers(0, m, (2000, 3))
    flat = (pick[:, 2] * m[1] + pick[:, 1]) * m[0] + pick[:, 0]
    for t in range(F):
        x = [fr[t, :, k].astype(np.float64) * float(grid.tpe[k]) for k in range(3)]
        c = np.ones(n)
        if window:
            c = np.prod([1 + np.cos(u) for u in x], 0) * 0.125
        ref = oracle.dirft_modes(x[0], x[1], x[2], c, -1, pick - m // 2)
        assert rel_l2(cs[t].ravel()[flat], ref) < 5 * eps + 3e-6, t


@pytest.mark.parametrize("centre", [(0.0, 0.0, 0.0), (1.0, 0.5, -0.25)])
@pytest.mark.parametrize("mask", [[1, 1, 1], [0, 1, 1], [0, 0, 0]])
def test_form_factors_and_masks(cuda, centre, mask):
    """X-ray weights at -k are those at k only on a centred Q grid.  FP32 at eps 1e-6 against FP64 at
    1e-10: FP32 rounding of the sums and of |Q|^2 in the exponentials (3e-5)."""
    rng = np.random.default_rng(5)
    fr = np.zeros((2, 900, 4), np.float32)
    fr[..., :3] = rng.uniform(-BOX / 2, BOX / 2, (2, 900, 3))
    grid = QGrid(_lib.BULK, (1, 1, 1), n_bz=20.25 * 2 * np.pi / BOX, a_par=(BOX,) * 3, ndim=3, q_center=centre)
    got = []
    for precision, eps in ((_lib.FP32, 1e-6), (_lib.FP64, 1e-10)):
        job = SqomJob(grid, species_counts=[500, 300, 100], n_frames=2, eps=eps, precision=precision,
                      weight_mode=_lib.WEIGHT_XRAY, xff=XFF, mask=mask)
        try:
            job.set_frames(fr)
            job.amplitudes_device().fill_(7.0)
            job.transform()
            got.append(job.amplitudes())
        finally:
            job.close()
    if not any(mask):
        assert not got[0].any() and not got[1].any()
    else:
        assert rel_l2(got[0], got[1]) < 3e-5
