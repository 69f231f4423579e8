"""The one-launch CG loop (k_cg_loop: f64 reductions, no multigrid) against the loop of separate kernels
(use_graphs = 0), at the sizes where it changes: one CTA and one cell, a partial CTA, every number of cells per
thread and its edges on 148 SMs x 512 threads, and a volume it leaves to the separate kernels.

Both run the same f32 operations per cell; only the order of the f64 partial sums differs, so alpha and
beta may differ by one f32 rounding (6e-8 relative) per iteration.  Over 12 iterations, each of which can
carry it into p once more, 12 * 2 * 6e-8 < 2e-6 of the largest pressure; the tolerance is 1e-5."""
import numpy as np
import pytest

from fluidisim_b200 import scenes
from fluidisim_b200.delta3d import Volume3

pytestmark = pytest.mark.gpu

ITERATIONS = 12


def volume(nx, ny, nz, bottom, graphs):
    dx = 0.1
    if bottom:  # a slope that the surface cuts: ghost faces with apertures other than 1
        i, j = np.meshgrid(np.arange(nx), np.arange(ny), indexing="xy")
        v = Volume3.configure_with_bottom(nx, ny, nz, dx, 1025.0, 9.81,
                                          (dx * nz * (0.05 + 0.6 * i / nx + 0.1 * j / ny)).astype(np.float32).ravel())
    else:
        v = Volume3.configure(nx, ny, nz, dx)
    v.set_options(use_graphs=graphs)
    rng = scenes.SplitMix64(7)
    eta = (dx * nz * (0.55 + 0.1 * rng.uniform_array(nx * ny, -1.0, 1.0))).astype(np.float32)
    v.set_free_surface(eta, float(np.float32(0.55 * dx * nz)))
    v.set_velocity(*[rng.uniform_array(n, -1.0, 1.0) for n in scenes.face_counts(nx, ny, nz)])
    return v


def compare(shape, bottom, linear):
    got = []
    for graphs in (1, 0):
        v = volume(*shape, bottom, graphs)
        call = v.project if linear else v.project_mobile3
        r = call(-1025.0 * 60.0, 1.0 / (1025.0 * 60.0), ITERATIONS)
        got.append((r, v.pressure(), v.velocity()))
        v.close()
    (a, pa, ua), (b, pb, ub) = got
    assert a.iterations == b.iterations
    assert np.abs(pa - pb).max() <= 1e-5 * max(np.abs(pb).max(), 1e-30)
    for x, y in zip(ua, ub):
        assert np.abs(x - y).max() <= 1e-5 * max(np.abs(y).max(), 1.0)
    return a


@pytest.mark.parametrize("linear", [False, True])
@pytest.mark.parametrize("bottom", [False, True])
@pytest.mark.parametrize("shape", [(3, 2, 4), (8, 8, 8), (33, 17, 5), (75, 61, 17), (76, 61, 33), (100, 64, 30),
                                   (101, 67, 40), (120, 99, 50), (128, 100, 70), (101, 101, 99)])
def test_one_launch_matches_the_separate_kernels(shape, bottom, linear):
    r = compare(shape, bottom, linear)
    assert 0 < r.iterations <= ITERATIONS


def test_larger_volumes_keep_the_separate_kernels():
    assert 148 * 512 * 12 < 101 * 101 * 99
    compare((101, 101, 99), False, False)


def test_nothing_to_solve():
    v = Volume3.configure(16, 8, 8, 0.1)
    rest = float(np.float32(0.45))
    v.set_free_surface(np.full(128, rest, np.float32), rest)
    r = v.project_mobile3(-1025.0 * 60.0, 1.0 / (1025.0 * 60.0))
    assert r.iterations == 0 and not v.pressure().any()


def test_concurrent_streams():
    """Cooperative launches from several host threads and streams: each waits until all of its CTAs fit."""
    from fluidisim_b200.batch import project_batch
    shapes = [(75, 61, 47), (64, 40, 33), (101, 67, 40), (31, 30, 29), (90, 81, 50), (75, 61, 47)]
    alone = []
    for s in shapes:
        v = volume(*s, False, 1)
        v.project_mobile3(-1025.0 * 60.0, 1.0 / (1025.0 * 60.0))
        alone.append(v.pressure())
        v.close()
    vols = [volume(*s, False, 1) for s in shapes]
    n = len(vols)
    reports, statuses = project_batch(vols, [-1025.0 * 60.0] * n, [1.0 / (1025.0 * 60.0)] * n, threads=n)
    assert statuses == [0] * n
    for v, p in zip(vols, alone):
        assert np.array_equal(v.pressure(), p)
        v.close()
