"""The one-launch multigrid loop (k_mg_loop, the default up to 2^20 cells) against the separate kernels of the same
march (kernels = 3), at the shapes where it changes: no coarse level, one, a large coarsest level without a tail, a tail
alone, levels above it, one tile and tiles cut by the edges, chunks of every height, FP16 storage, a sparse set.

Both run the same f32 operations per cell; only the order of the f64 partial sums differs, so alpha and beta
may differ by one f32 rounding (6e-8 relative) per iteration.  Over 8 iterations 8 * 2 * 6e-8 = 1e-6 of the largest
pressure; FP16 storage rounds at 5e-4 what such a change moves across a rounding boundary.  Tolerances 1e-5 and 1e-3."""
import numpy as np
import pytest

from fluidisim_b200 import scenes
from fluidisim_b200.delta3d import STORAGE_F16, Volume3

pytestmark = pytest.mark.gpu

SCALE, K1 = -1025.0 * 60.0, 1.0 / (1025.0 * 60.0)


def volume(shape, kernels, storage=0, sparse=False, levels=0):
    nx, ny, nz = shape
    dx = 0.1
    i, j = np.meshgrid(np.arange(nx), np.arange(ny), indexing="xy")
    bottom = (0.1 * dx * nz * (1.0 + np.sin(5.0 * i / nx) * np.cos(4.0 * j / ny))).astype(np.float32)
    v = Volume3.configure_with_bottom(nx, ny, nz, dx, 1025.0, 9.81, bottom.ravel())
    v.set_options(kernels=kernels, storage=storage, mg_max_levels=levels)
    v.enable_multigrid()
    rest = float(np.float32(0.6 * nz * dx))
    mask = np.ones((ny, nx), bool)
    if sparse:
        mask[:, : nx // 2] = False
        v.set_free_surface(np.full(nx * ny, rest, np.float32), rest)
        v.enable_sparse()
        v.set_active_columns(mask)
    eta = np.where(mask, rest + 0.2 * nz * dx * np.sin(7.0 * i / nx + 3.0 * j / ny), np.float32(rest))
    v.set_free_surface(eta.astype(np.float32).ravel(), rest)
    rng = scenes.SplitMix64(5)
    v.set_velocity(*[rng.uniform_array(n, -1.0, 1.0) for n in scenes.face_counts(nx, ny, nz)])
    return v


def compare(shape, iterations=8, tolerance=1e-5, **kw):
    got = []
    for kernels in (0, 3):
        v = volume(shape, kernels, **kw)
        r = v.project_mobile3(SCALE, K1, iterations)
        got.append((r, v.pressure(), v.velocity()))
        v.close()
    (a, pa, ua), (b, pb, ub) = got
    assert a.iterations == b.iterations
    assert np.abs(pa - pb).max() <= tolerance * np.abs(pb).max()
    for x, y in zip(ua, ub):
        assert np.abs(x - y).max() <= tolerance * max(np.abs(y).max(), 1.0)


@pytest.mark.parametrize("shape", [(4, 4, 4), (6, 5, 7), (8, 8, 8), (16, 16, 16), (34, 10, 22), (30, 30, 30), (66, 40, 50),
                                   (64, 64, 64), (64, 8, 8), (8, 64, 32), (130, 36, 12), (96, 96, 96), (128, 128, 64)])
def test_one_launch_matches_the_separate_kernels(shape):
    compare(shape)


@pytest.mark.parametrize("kw", [dict(storage=STORAGE_F16, tolerance=1e-3), dict(sparse=True), dict(levels=1),
                                dict(levels=2), dict(iterations=1)])
def test_options(kw):
    compare((64, 48, 32), **kw)


def test_runs_repeat_and_converge():
    """The same call twice gives the same bits (the sums have a fixed order), and meets the acceptance."""
    out = []
    for _ in range(2):
        v = volume((80, 64, 48), 0)
        r = v.project_mobile3(SCALE, K1)
        assert not r.degraded and r.residual <= 1e-6
        out.append((r, v.pressure()))
        v.close()
    assert out[0][0] == out[1][0] and np.array_equal(out[0][1], out[1][1])


def test_concurrent_streams():
    from fluidisim_b200.batch import project_batch
    shapes = [(32, 32, 32), (64, 48, 32), (48, 48, 48), (16, 16, 16), (64, 64, 64), (34, 10, 22)]
    alone = []
    for s in shapes:
        v = volume(s, 0)
        v.project_mobile3(SCALE, K1)
        alone.append(v.pressure())
        v.close()
    vols = [volume(s, 0) for s in shapes]
    _, statuses = project_batch(vols, [SCALE] * len(vols), [K1] * len(vols), threads=len(vols))
    assert statuses == [0] * len(vols)
    for v, p in zip(vols, alone):
        assert np.array_equal(v.pressure(), p)
        v.close()
