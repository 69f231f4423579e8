"""A volume whose row records find no memory is configured without them and gives the same bits: the GPU is filled so that
the records do not fit, at the configuration, or when the multigrid's arrays need their place.  And small volumes hold
what they use: a batch configures hundreds of them."""
import numpy as np
import pytest

from fluidisim_b200 import scenes
from fluidisim_b200.delta3d import Volume3

pytestmark = pytest.mark.gpu

SHAPE = (128, 128, 128)
RECORDS = 32 * 128 ** 3  # bytes
SCALE, K1 = -1025.0 * 60.0, 1.0 / (1025.0 * 60.0)


def configure():
    nx, ny, nz = SHAPE
    i, j = np.meshgrid(np.arange(nx), np.arange(ny), indexing="xy")
    return Volume3.configure_with_bottom(nx, ny, nz, 0.1, 1025.0, 9.81, (0.8 + 0.5 * np.sin(9.0 * i / nx + 5.0 * j / ny))
                                         .astype(np.float32).ravel())


def project(v):
    nx, ny, nz = SHAPE
    i, j = np.meshgrid(np.arange(nx), np.arange(ny), indexing="xy")
    rest = float(np.float32(7.0))
    v.set_free_surface((rest + 0.4 * np.sin(7.0 * i / nx + 3.0 * j / ny)).astype(np.float32).ravel(), rest)
    rng = scenes.SplitMix64(5)
    v.set_velocity(*[rng.uniform_array(n, -1.0, 1.0) for n in scenes.face_counts(*SHAPE)])
    return v.project_mobile3(SCALE, K1, 12), v.pressure()


@pytest.mark.parametrize("when", ["configure", "multigrid"])
def test_a_volume_without_room_for_its_records(when):
    import torch

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    torch.cuda.empty_cache()
    start = free()
    v = configure()
    configured = free()
    v.enable_multigrid()
    whole = free()
    want = project(v)
    v.close()
    need = start - (configured if when == "configure" else whole)  # with the records
    fill = torch.empty(free() - need + RECORDS // 2, dtype=torch.uint8, device="cuda")
    try:
        w = configure()
        if when == "configure":  # the multigrid's arrays find their place again
            del fill
            torch.cuda.empty_cache()
        w.enable_multigrid()
        got = project(w)
        w.close()
    finally:
        fill = None
        torch.cuda.empty_cache()
    assert got[0] == want[0] and np.array_equal(got[1], want[1])


def test_small_volumes_hold_what_they_use():
    """64 volumes of 16^3 cells with cut cells and hierarchy: 128 B a cell of fields (32 floats), 32 of records and 23 of
    coarse levels, 0.75 MB; twice that is the bound (a chunk of 4 MB each was 4.2)."""
    import torch
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    volumes = [Volume3.configure_with_bottom(16, 16, 16, 0.1, 1025.0, 9.81, np.full(256, 0.1, np.float32)) for _ in range(64)]
    for v in volumes:
        v.enable_multigrid()
    torch.cuda.synchronize()
    each = (before - torch.cuda.mem_get_info()[0]) / 64
    for v in volumes:
        v.close()
    assert each < 1.5e6
