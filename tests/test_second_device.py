"""Jobs on a second device of one process: every kernel that takes more than 48 KB of dynamic shared memory
has to ask for it on each device (stand-in runtime, no GPU)."""
import fake_cuda

PROGRAM = r"""
def jobs():
    for precision, ndim, repro in ((_lib.FP32, 2, 0), (_lib.FP64, 2, 0), (_lib.FP32, 3, 0), (_lib.FP32, 3, 1),
                                   (_lib.FP64, 3, 0)):
        grid = QGrid(_lib.BULK, (1, 1, 1), n_bz=20.25 * 2 * np.pi / 20.0, a_par=(20.0,) * 3, ndim=ndim)
        for eps in (1e-3, 1e-7):
            job = SqomJob(grid, species_counts=[300, 200, 100], n_frames=9, precision=precision, eps=eps)
            job.set_option(_lib.OPT_REPRODUCIBLE, repro)
            job.set_frames(np.zeros((9, 600, 4), np.float32))
            job.transform()
            job.sq_total()
            ta = TimeAxis(9, 0.01)
            job.sqw_econst(ta, 1)
            job.sqw_dispersion(ta, np.arange(4))
            job.iqt(ta.n_int, 1)
            job.close()

for device in (0, 1):
    fake.fake_set_device(device)
    n = fake.fake_launches()
    jobs()
    print(device, fake.fake_launches() - n)
assert fake.fake_held() == 0
"""


def test_large_shared_memory_is_asked_for_on_each_device(lib, tmp_path):
    out = [line.split() for line in fake_cuda.run(tmp_path, PROGRAM).splitlines()]
    assert out[0][1] == out[1][1] and int(out[0][1]) > 100
