"""A recorded choice of the tuner is not taken by a job that runs its frames differently: the z-slab pipeline
tuned on a job of one frame would switch the frame batches of a longer run off (stand-in runtime)."""
import fake_cuda

PROGRAM = r"""
def lines():
    return [l.split()[0] for l in open(cache)]

def tune(frames, **kw):
    grid = QGrid(_lib.BULK, (1, 1, 1), n_bz=40.25 * 2 * np.pi / 20.0, a_par=(20.0,) * 3, ndim=3)
    job = SqomJob(grid, species_counts=[300, 200], n_frames=frames, eps=1e-5, stream_ordered=True, **kw)
    job.set_frames(np.zeros((frames, 500, 4), np.float32))
    job.autotune(0, frames, cache=cache)
    job.close()
    return len(lines())

print(tune(1), tune(1), tune(16), tune(16), tune(16, frame_batch=False), len(set(lines())))
"""


def test_choices_of_one_frame_and_of_batches_are_kept_apart(lib, tmp_path):
    out = fake_cuda.run(tmp_path, f"cache = {str(tmp_path / 'tune.txt')!r}\n" + PROGRAM)
    assert out.split() == ["1", "1", "2", "2", "2", "2"]
