"""Which loop a projection runs, by its launches: a one-launch loop is one launch whatever the iterations, the separate
kernels are four an iteration without the multigrid and more with it.  Other tests compare results between the routes;
these fail when both sides run the same one."""
import numpy as np
import pytest

from fluidisim_b200 import scenes
from fluidisim_b200.delta3d import STORAGE_F16, Volume3

pytestmark = pytest.mark.gpu

SCALE, K1 = -1025.0 * 60.0, 1.0 / (1025.0 * 60.0)
SETUP = 40  # launches of a projection outside its loops: set-up, checks and publishing of up to four outer iterations


def launches(shape, multigrid, linear=False, iterations=12, **options):
    nx, ny, nz = shape
    v = Volume3.configure(nx, ny, nz, 0.1, 1025.0, 9.81)
    v.set_options(**options)
    if multigrid:
        v.enable_multigrid()
    rest = float(np.float32(0.055 * nz))
    v.set_free_surface(np.full(nx * ny, rest, np.float32), rest)
    rng = scenes.SplitMix64(5)
    v.set_velocity(*[rng.uniform_array(n, -1.0, 1.0) for n in scenes.face_counts(nx, ny, nz)])
    before = v.kernel_launches()
    r = (v.project if linear else v.project_mobile3)(SCALE, K1, iterations)
    n = v.kernel_launches() - before
    v.close()
    assert r.iterations >= 8
    return n, r.iterations


@pytest.mark.parametrize("storage", [0, STORAGE_F16])
@pytest.mark.parametrize("shape", [(32, 16, 24), (64, 64, 64), (128, 64, 48)])
def test_multigrid_in_one_launch_up_to_the_line(shape, storage):
    n, its = launches(shape, True, storage=storage)
    assert n <= SETUP
    n, its = launches(shape, True, kernels=3, storage=storage)
    assert n >= 6 * its


def test_without_a_coarse_level_the_line_is_higher():
    assert launches((124, 62, 93), True)[0] <= SETUP
    n, its = launches((102, 101, 102), True)
    assert 102 * 101 * 102 > 2 ** 20 and n >= 6 * its


@pytest.mark.parametrize("shape", [(130, 64, 48), (72, 72, 80)])
def test_multigrid_above_the_line(shape):
    assert 3 * 2 ** 17 < shape[0] * shape[1] * shape[2]
    n, its = launches(shape, True)
    assert n >= 6 * its
    assert n == launches(shape, True, kernels=3)[0]


@pytest.mark.parametrize("linear", [False, True])
def test_without_the_multigrid(linear):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n, its = launches((31, 30, 29), False, linear)
    assert n <= SETUP
    n, its = launches((31, 30, 29), False, linear, use_graphs=0)
    assert n >= 4 * its
    side = 101
    layers = sms * 512 * 12 // (side * side) + 1  # the first that its threads do not hold
    n, its = launches((side, side, layers), False, linear)
    assert n >= 4 * its
    n, its = launches((side, side, layers - 1), False, linear)
    assert n <= SETUP


def test_ordered_sums_and_host_loops_keep_the_separate_kernels():
    for options in (dict(reduction=1), dict(use_graphs=0)):
        n, its = launches((32, 32, 32), True, **options)
        assert n >= 6 * its
