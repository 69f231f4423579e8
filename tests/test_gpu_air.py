"""Projections that leave the air above the surface alone, against the same with every layer processed
(no_tile_skip = 1): a skipped cell holds 0 and adds 0, so pressure, velocities and report are the same bits.
One volume runs a sequence of surfaces, falling and rising across the tiles' and chunks' edges, so that a vector
left over from a higher surface would show; and a refused projection in between, whose vectors are not finite."""
import numpy as np
import pytest

from fluidisim_b200 import scenes
from fluidisim_b200.delta3d import Delta3dError, STORAGE_F16, Volume3

pytestmark = pytest.mark.gpu

SCALE, K1 = -1025.0 * 60.0, 1.0 / (1025.0 * 60.0)
# surface height (share of the depth) and swing of each projection of a sequence
SURFACES = [(0.85, 0.1), (0.3, 0.05), (0.55, 0.35), (0.12, 0.02), (0.97, 0.0)]


def run(shape, skip, refused=False, storage=0, kernels=0, sparse=False):
    nx, ny, nz = shape
    dx = 0.1
    rng = scenes.SplitMix64(11)
    sdf = scenes.spheres_sdf(nx, ny, nz, dx, [(0.3 * nx * dx, 0.5 * ny * dx, 0.3 * nz * dx)], [0.15 * min(shape) * dx])
    v = Volume3.configure_with_solid(nx, ny, nz, dx, 1025.0, 9.81, np.zeros(nx * ny, np.float32), sdf)
    v.set_options(no_tile_skip=0 if skip else 1, storage=storage, kernels=kernels)
    v.enable_multigrid()
    mask = np.ones((ny, nx), bool)
    if sparse:
        mask[:, nx // 2:] = False
        v.set_free_surface(np.full(nx * ny, 0.5, np.float32), 0.5)
        v.enable_sparse()
        v.set_active_columns(mask)
    i, j = np.meshgrid(np.arange(nx), np.arange(ny), indexing="xy")
    out = []
    for q, (level, swing) in enumerate(SURFACES):
        h = nz * dx * (level + swing * np.sin(6.0 * i / nx + 3.0 * j / ny + q))
        rest = np.float32(0.5) if sparse else np.float32(level * nz * dx)
        eta = np.where(mask, np.clip(h, 0.05, nz * dx * 0.999), rest).astype(np.float32)
        v.set_free_surface(eta.ravel(), float(rest))
        vel = [rng.uniform_array(n, -1.0, 1.0) for n in scenes.face_counts(nx, ny, nz)]
        if refused and q % 2 == 0:
            v.set_velocity(*[f * np.float32(3e37) for f in vel])
            with pytest.raises(Delta3dError):
                v.project_mobile3(SCALE, K1)
        v.set_velocity(*vel)
        r = v.project_mobile3(SCALE, K1, 40)
        out.append((r, v.pressure(), *v.velocity()))
    v.close()
    return out


def same(a, b):
    for (ra, *fa), (rb, *fb) in zip(a, b):
        assert ra == rb
        for x, y in zip(fa, fb):
            assert np.array_equal(x, y)


@pytest.mark.parametrize("shape", [(16, 16, 16), (34, 10, 22), (64, 8, 8), (72, 24, 40), (96, 40, 64), (130, 66, 12)])
def test_air_is_left_alone(shape):
    same(run(shape, True), run(shape, False))


@pytest.mark.parametrize("kw", [dict(storage=STORAGE_F16), dict(kernels=5), dict(kernels=4), dict(kernels=2),
                                dict(sparse=True), dict(refused=True), dict(refused=True, kernels=5)])
def test_air_in_every_family(kw):
    same(run((64, 24, 32), True, **kw), run((64, 24, 32), False, **kw))


def test_a_step_after_a_refusal():
    """The step's check of every work vector sees none of a refused projection's values in the air."""
    v = Volume3.configure(32, 16, 24, 0.1)
    v.enable_multigrid()
    high, low = (np.full(512, np.float32(x), np.float32) for x in (2.1, 0.8))
    rng = scenes.SplitMix64(3)
    vel = [rng.uniform_array(n, -1.0, 1.0) for n in scenes.face_counts(32, 16, 24)]
    v.set_free_surface(high, 2.1)
    v.set_velocity(*[f * np.float32(3e37) for f in vel])
    with pytest.raises(Delta3dError):
        v.project_mobile3(SCALE, K1)
    v.set_free_surface(low, 0.8)
    v.set_velocity(*[np.float32(0.01) * f for f in vel])
    v.step_surface_mobile(2000)
