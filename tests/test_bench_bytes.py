"""The bench line's algorithmic bytes: a pass that leaves the air alone is counted with the layers it visits."""
import numpy as np

import bench


def scene(nx, ny, nz, eta, dx=0.1):
    return dict(nx=nx, ny=ny, nz=nz, dx=np.float32(dx), eta=np.asarray(eta, np.float32).ravel())


def test_a_flat_surface():
    s = scene(64, 16, 20, np.full((16, 64), 0.86))  # nine layers have their centre below 0.86 m: ten are marched
    assert bench.marched_cells(s) == 64 * 16 * 10
    assert bench.alg_bytes_per_launch("kx_update_rn", s) == 24 * 64 * 16 * 10
    assert bench.alg_bytes_per_launch("kt_dir_apply_dot", s) == 18 * 64 * 16 * 10
    assert bench.alg_bytes_per_launch("kz_fine_pre", s) == 14 * 64 * 16 * 20  # a family that visits every layer


def test_each_tile_up_to_its_highest_column():
    rng = np.random.default_rng(3)
    nx, ny, nz = 100, 20, 31
    eta = rng.uniform(-0.2, 3.3, (ny, nx)).astype(np.float32) * np.where(np.arange(nx) < 64, np.float32(0.3), np.float32(1.0))
    want = 0
    for j in range(0, ny, 8):
        for i in range(0, nx, 64):
            tile = eta[j:j + 8, i:i + 64]
            top = max(sum((np.float32(k) + np.float32(0.5)) * np.float32(0.1) < h for k in range(nz)) for h in tile.ravel())
            want += tile.size * min((top + 1) // 2 * 2, nz)
    assert bench.marched_cells(scene(nx, ny, nz, eta)) == want


def test_every_pass_of_the_default_paths_has_its_bytes():
    for name in ("kx_update_rn", "kx_residual", "k_rhs_march", "kx_fine_pre", "kt_fine_post1", "kt_residual"):
        assert bench.BYTES_PER_CELL[name] > 0
