"""mp_sql's one-call jobs leave the process's memory pools alone and little memory behind."""
import gc

import numpy as np
import pytest

import fake_cuda
from mp_tools_gb300 import sql

PROGRAM = r"""
from mp_tools_gb300 import sql
fr = np.random.default_rng(1).uniform(-10, 10, (2, 600, 4)).astype(np.float32)
sql.transform_histogram(fr, [400, 200], sql.SqlGrid(3.0, (20.0,) * 3), 0.05, eps=1e-5)
print(fake.fake_default_threshold(0), fake.fake_held())
"""


def test_the_default_pool_keeps_its_release_threshold(lib, tmp_path):
    assert fake_cuda.run(tmp_path, PROGRAM).split() == ["0", "0"]


@pytest.mark.gpu
def test_memory_left_after_calls(lib, cuda):
    """Jobs of about 0.5 GB: at most 512 MB stay for the next call, and mpsq_release_memory gives them back
    (up to 32 MB that kernels loaded meanwhile may hold)."""
    fr = np.zeros((1, 30000, 4), np.float32)
    fr[..., :3] = np.random.default_rng(1).uniform(-39, 39, (1, 30000, 3))
    grid = sql.SqlGrid(6.0, (79.4,) * 3)
    small = sql.SqlGrid(1.0, (79.4,) * 3)
    sql.transform_histogram(fr, [28000, 2000], small, 0.01)        # loads the kernels
    lib.mpsq_release_memory()
    gc.collect()
    cuda.cuda.synchronize()
    free = cuda.cuda.mem_get_info()[0]
    want = sql.transform_histogram(fr, [28000, 2000], grid, 0.01)
    for _ in range(3):
        assert np.allclose(sql.transform_histogram(fr, [28000, 2000], grid, 0.01), want, rtol=1e-4, atol=1e-9)
    cuda.cuda.synchronize()
    assert free - cuda.cuda.mem_get_info()[0] <= (512 + 32) << 20
    lib.mpsq_release_memory()
    assert free - cuda.cuda.mem_get_info()[0] <= 32 << 20


@pytest.mark.gpu
def test_calls_from_several_threads(lib, cuda):
    """Threads share the pool; each gets the histogram of its own frames."""
    import threading
    rng = np.random.default_rng(2)
    frames = [np.zeros((1, 3000, 4), np.float32) for _ in range(6)]
    for fr in frames:
        fr[..., :3] = rng.uniform(-10, 10, (1, 3000, 3))
    grid = sql.SqlGrid(5.0, (20.0,) * 3)
    want = [sql.transform_histogram(fr, [2000, 1000], grid, 0.05) for fr in frames]
    got = [None] * 6

    def work(i):
        stream = cuda.cuda.Stream()
        for _ in range(5):
            got[i] = sql.transform_histogram(frames[i], [2000, 1000], grid, 0.05, stream=stream.cuda_stream)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(6)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    for g, w in zip(got, want):
        assert np.allclose(g, w, rtol=1e-4, atol=1e-6 * np.abs(w).max())
