"""The marching assembly where it zeroes the loop's vectors (the multigrid, f64 sums: the air is left alone) against the
pass of one cell per thread of the ordered sums, which visits every cell.  One volume takes a high surface and then
lower ones, so that what the march failed to zero would be the former projection's values.

The rows are the same f32 operations, so three iterations differ by the sums alone: an f32 sum of n products in
chunks of 64 is within (64 + n / 64) 6e-8 of the f64 one, at most 1.6e-5 for the 13,000 cells here, and three
iterations take six of them: 1e-4 of the largest pressure."""
import numpy as np
import pytest

from fluidisim_b200 import scenes
from fluidisim_b200.delta3d import Volume3

pytestmark = pytest.mark.gpu

SCALE, K1 = -1025.0 * 60.0, 1.0 / (1025.0 * 60.0)


def project(shape, kind, reduction, kernels):
    nx, ny, nz = shape
    dx = 0.1
    sdf = scenes.spheres_sdf(nx, ny, nz, dx, [(0.4 * nx * dx, 0.5 * ny * dx, 0.2 * nz * dx)], [0.12 * min(shape) * dx])
    if kind == "flat":
        v = Volume3.configure(nx, ny, nz, dx, 1025.0, 9.81)
    else:
        v = Volume3.configure_with_solid(nx, ny, nz, dx, 1025.0, 9.81, np.zeros(nx * ny, np.float32), sdf)
    if kind == "moving":
        v.set_solid_rigid(sdf, (0.2, -0.1, 0.3), (0.0, 0.5, 0.1), (0.4 * nx * dx, 0.5 * ny * dx, 0.2 * nz * dx))
    v.set_options(reduction=reduction, kernels=kernels)
    v.enable_multigrid()
    mask = np.ones((ny, nx), bool)
    if kind == "sparse":
        mask[:, nx // 2:] = False
        rest = np.float32(0.5 * nz * dx)
        v.set_free_surface(np.full(nx * ny, rest, np.float32), float(rest))
        v.enable_sparse()
        v.set_active_columns(mask)
    i, j = np.meshgrid(np.arange(nx), np.arange(ny), indexing="xy")
    rng = scenes.SplitMix64(13)
    out = []
    for level, swing in ((0.85, 0.1), (0.5, 0.3), (0.35, 0.02)):
        rest = np.float32((0.5 if kind == "sparse" else level) * nz * dx)
        eta = nz * dx * (level + swing * np.sin(6.0 * i / nx + 3.0 * j / ny))
        v.set_free_surface(np.where(mask, eta, rest).astype(np.float32).ravel(), float(rest))
        v.set_velocity(*[rng.uniform_array(n, -1.0, 1.0) for n in scenes.face_counts(nx, ny, nz)])
        v.project_mobile3(SCALE, K1, 3)
        out.append(v.pressure())
    v.close()
    return out


@pytest.mark.parametrize("kernels", [0, 3])
@pytest.mark.parametrize("kind", ["flat", "cut", "sparse", "moving"])
@pytest.mark.parametrize("shape", [(32, 8, 8), (34, 10, 18), (64, 16, 12), (100, 4, 30)])
def test_march_zeroes_what_the_pass_per_cell_writes(shape, kind, kernels):
    for a, b in zip(project(shape, kind, 0, kernels), project(shape, kind, 1, 0)):
        assert np.abs(b).max() > 0.0
        assert np.abs(a - b).max() <= 1e-4 * np.abs(b).max()
