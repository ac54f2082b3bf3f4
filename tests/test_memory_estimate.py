"""mpsq_job_estimate_bytes covers the device memory that a job takes, frame batches included, and a
server's budget covers its jobs (stand-in runtime that keeps account, no GPU)."""
import fake_cuda

JOBS = r"""
import itertools
for precision, ndim, F, edge, n in itertools.product((_lib.FP32, _lib.FP64), (2, 3), (1, 2, 5, 40), (6.25, 24.25, 60.25),
                                                     (700, 30000)):
    if ndim == 3 and edge > 40:
        continue
    for store, window, ordered, centre, batch in ((0, 0, 0, 0, 1), (F < 6, 1, 1, 0, 1), (0, 0, 1, 1, 1), (0, 1, 0, 1, 1),
                                                  (0, 0, 1, 0, 0)):
        grid = QGrid(_lib.BULK, (1, 1, 1), n_bz=edge * 2 * np.pi / 20.0, a_par=(20.0,) * 3, ndim=ndim,
                     q_center=(float(centre), 0.0, 0.0))
        kw = dict(species_counts=[n // 2, n // 3, n - n // 2 - n // 3], n_frames=F, precision=precision, eps=1e-6,
                  store_species=bool(store), window=bool(window), stream_ordered=bool(ordered), frame_batch=bool(batch))
        est = SqomJob.estimate_bytes(SqomJob.describe(grid, **kw))
        before = fake.fake_held()
        fake.fake_most(1)
        job = SqomJob(grid, **kw)
        job.set_frames(np.zeros((F, n, 4), np.float32))
        job.transform()
        most = fake.fake_most(1) - before
        job.close()
        assert fake.fake_held() == before
        print(precision, ndim, F, batch, most, est, "short" if most > est else "ok", *kw.items())
"""

SERVER = r"""
import torch
from mp_tools_gb300 import serve
rng = np.random.default_rng(3)
ex = serve.GpuExecutor()
reqs = [serve.abo3_request(i, 0.0, 6, 24, 3, rng, pinned=False) for i in range(3)]
for budget in (int(2.5 * ex._bytes(reqs[0], 0)), 40 << 30):
    ex.budget, ex.max_active = budget, 2
    promised, jobs = 0, []
    before = fake.fake_held()
    for r in reqs[:2]:
        b = ex.estimate(r)
        assert b <= budget and r._q_slab == 0, (b, budget)
        d = ex._describe(r, r._q_slab, r._frame_batch)
        promised += b
        jobs.append(SqomJob(r.grid, species_counts=r.counts, n_frames=24, stream_ordered=True, frame_batch=r._frame_batch,
                            **r.job_kwargs))
    assert fake.fake_held() - before <= promised <= budget, (fake.fake_held(), promised, budget)
    print(reqs[0]._frame_batch)
    for j in jobs:
        j.close()
"""


def test_estimate_covers_creation_and_transform(lib, tmp_path):
    rows = fake_cuda.run(tmp_path, JOBS).splitlines()
    assert len(rows) > 200
    assert not [r for r in rows if " short " in r]
    # every kind of job takes batches where it has frames for them, and leaves them out on request
    most = {}
    for r in rows:
        p, ndim, F, batch, held, est = r.split()[:6]
        most.setdefault((p, ndim, F, batch), []).append(int(held))
    for p, ndim in (("0", "2"), ("0", "3"), ("1", "2"), ("1", "3")):
        assert max(most[p, ndim, "40", "1"]) > 2 * max(most[p, ndim, "40", "0"]), (p, ndim)


def test_a_small_budget_covers_its_jobs(lib, tmp_path):
    """Two jobs that fit a budget without batches are admitted together and stay within it; a large
    budget lets them take their batches."""
    assert fake_cuda.run(tmp_path, SERVER).split() == ["False", "True"]


MAPS = r"""
import threading
for precision, ndim, ordered, store in ((_lib.FP32, 2, 0, 0), (_lib.FP64, 2, 0, 1), (_lib.FP32, 3, 0, 0), (_lib.FP32, 3, 1, 1)):
    grid = QGrid(_lib.BULK, (1, 1, 1), n_bz=(700.25 if ndim == 2 else 60.25) * 2 * np.pi / 20.0, a_par=(20.0,) * 3, ndim=ndim)
    kw = dict(species_counts=[400, 300], n_frames=8, precision=precision, eps=1e-3, store_species=bool(store),
              stream_ordered=bool(ordered))
    est = SqomJob.estimate_bytes(SqomJob.describe(grid, **kw))
    before = fake.fake_held()
    job = SqomJob(grid, **kw)
    created = fake.fake_held() - before
    ta, q2 = TimeAxis(8, 0.01), np.ones(grid.n_modes, np.float32)
    for _ in range(2):
        job.sq_total()
        job.sqw_econst(ta, 1, q2_norm=q2)
        job.sqw_dispersion(ta, np.arange(grid.n_modes, dtype=np.int64) % 50)
        job.iqt(ta.n_int, 1, q2_norm=q2)
        job.iqt_dispersion(ta.n_int, np.arange(30))
        job.sqw_gauss(q2_norm=q2)
        if store:
            job.radial_hist(np.eye(3), np.asarray(grid.tpe, np.float64), 0.1, 4.0, 40)
    held = fake.fake_held() - before
    threads = [threading.Thread(target=job.sqw_econst, args=(ta, 1)) for _ in range(6)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert fake.fake_held() - before == held
    print(created, held, est)
    job.close()
    assert fake.fake_held() == before
"""


def test_estimate_covers_what_map_calls_leave(lib, tmp_path):
    """A plain job keeps buffers of its map calls within its estimate, a stream-ordered one none."""
    rows = [[int(v) for v in r.split()] for r in fake_cuda.run(tmp_path, MAPS).splitlines()]
    assert len(rows) == 4 and all(held <= est for _, held, est in rows)
    assert rows[0][1] > rows[0][0] and rows[3][1] == rows[3][0]
