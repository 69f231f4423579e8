"""A one-launch loop whose grid-wide meeting does not complete gives up, says why, leaves the volume as it was and usable.
The meeting is made to wait for a block that does not exist; each block polls a bounded number of times and returns."""
import time

import numpy as np
import pytest

from fluidisim_b200 import scenes
from fluidisim_b200.batch import project_batch
from fluidisim_b200.delta3d import Delta3dError, STORAGE_F16, Volume3, library

pytestmark = pytest.mark.gpu

SCALE, K1 = -1025.0 * 60.0, 1.0 / (1025.0 * 60.0)


def volume(multigrid, storage=0):
    shape = (32, 16, 24)
    v = Volume3.configure(*shape, 0.1, 1025.0, 9.81)
    v.set_options(storage=storage)
    if multigrid:
        v.enable_multigrid()
    v.set_free_surface(np.full(512, np.float32(1.4), np.float32), 1.4)
    rng = scenes.SplitMix64(5)
    v.set_velocity(*[rng.uniform_array(n, -1.0, 1.0) for n in scenes.face_counts(*shape)])
    return v


@pytest.mark.parametrize("kind", ["multigrid", "f16", "jacobi", "linear"])
def test_a_meeting_that_runs_out(kind):
    v = volume(kind in ("multigrid", "f16"), STORAGE_F16 if kind == "f16" else 0)
    call = v.project if kind == "linear" else v.project_mobile3
    before = [v.pressure(), *v.velocity()]
    assert library().fd3_absent_blocks_for_tests(v._h, 1) == 0
    t = time.perf_counter()
    with pytest.raises(Delta3dError) as e:
        call(SCALE, K1)
    t = time.perf_counter() - t
    assert e.value.kind == "Cuda" and "meeting" in str(e.value)
    assert 0.05 < t < 10.0
    for a, b in zip(before, [v.pressure(), *v.velocity()]):
        assert np.array_equal(a, b)
    assert library().fd3_absent_blocks_for_tests(v._h, 0) == 0
    r = call(SCALE, K1)
    w = volume(kind in ("multigrid", "f16"), STORAGE_F16 if kind == "f16" else 0)
    assert r == (w.project if kind == "linear" else w.project_mobile3)(SCALE, K1)
    assert np.array_equal(v.pressure(), w.pressure())


def test_a_batch_hands_the_reason_to_its_caller():
    vols = [volume(True), volume(False)]
    library().fd3_absent_blocks_for_tests(vols[1]._h, 1)
    _, statuses = project_batch(vols, [SCALE] * 2, [K1] * 2, threads=2)
    assert statuses == [0, 100]
    assert b"meeting" in library().fd3_last_cuda_error()
