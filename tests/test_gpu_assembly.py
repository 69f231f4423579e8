"""The assembly that marches the columns (k_rhs_march, the default with f64 sums) against the pass of one cell per
thread (k_rhs_b2, which the ordered sums keep), at volumes cut by its tiles' and blocks' edges, on a flat bottom,
with cut cells, a sparse set and a moving solid, with the air left alone and not.

The rows are the same f32 operations, so three iterations from p = 0 differ by the sums alone: an f32 sum of n
products in chunks of 64 is within (64 + n / 64) 6e-8 of the f64 one, at most 1.6e-5 for the 13,000 cells here, and
three iterations take six of them: 1e-4 of the largest pressure."""
import numpy as np
import pytest

from fluidisim_b200 import scenes
from fluidisim_b200.delta3d import Volume3

pytestmark = pytest.mark.gpu

SCALE, K1 = -1025.0 * 60.0, 1.0 / (1025.0 * 60.0)
ORDERED = 1


def project(shape, kind, reduction):
    nx, ny, nz = shape
    dx = 0.1
    rng = scenes.SplitMix64(13)
    sdf = scenes.spheres_sdf(nx, ny, nz, dx, [(0.4 * nx * dx, 0.5 * ny * dx, 0.4 * nz * dx)], [0.2 * min(shape) * dx])
    if kind == "flat":
        v = Volume3.configure(nx, ny, nz, dx, 1025.0, 9.81)
    else:
        v = Volume3.configure_with_solid(nx, ny, nz, dx, 1025.0, 9.81, np.zeros(nx * ny, np.float32), sdf)
    if kind == "moving":
        v.set_solid_rigid(sdf, (0.2, -0.1, 0.3), (0.0, 0.5, 0.1), (0.4 * nx * dx, 0.5 * ny * dx, 0.4 * nz * dx))
    v.set_options(reduction=reduction, no_tile_skip=1 if kind == "all layers" else 0)
    rest = np.float32(0.6 * nz * dx)
    mask = np.ones((ny, nx), bool)
    if kind == "sparse":
        mask[:, nx // 2:] = False
        v.set_free_surface(np.full(nx * ny, rest, np.float32), float(rest))
        v.enable_sparse()
        v.set_active_columns(mask)
    i, j = np.meshgrid(np.arange(nx), np.arange(ny), indexing="xy")
    eta = rest + 0.3 * nz * dx * np.sin(6.0 * i / nx + 3.0 * j / ny)
    v.set_free_surface(np.where(mask, eta, rest).astype(np.float32).ravel(), float(rest))
    v.set_velocity(*[rng.uniform_array(n, -1.0, 1.0) for n in scenes.face_counts(nx, ny, nz)])
    v.project_mobile3(SCALE, K1, 3)
    p = v.pressure()
    v.close()
    return p


@pytest.mark.parametrize("kind", ["flat", "cut", "sparse", "moving", "all layers"])
@pytest.mark.parametrize("shape", [(32, 8, 8), (33, 9, 17), (64, 16, 12), (5, 70, 6), (100, 4, 30)])
def test_march_matches_the_pass_per_cell(shape, kind):
    a, b = project(shape, kind, 0), project(shape, kind, ORDERED)
    assert np.abs(b).max() > 0.0
    assert np.abs(a - b).max() <= 1e-4 * np.abs(b).max()
