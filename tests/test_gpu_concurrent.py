"""Volumes projected at once run side by side, and each has the bits it has alone.

The one-launch loops (k_mg_loop, k_cg_loop) keep their SMs for a whole solve: with every SM each, volumes on several
streams followed one another, in 0.88 to 0.92 of the time of one worker (two threads: about 1).  Now eight workers have
eight volumes done in 0.2 to 0.6 of it and two threads two in 0.5 to 0.65; the bounds lie between."""
import threading
import time

import numpy as np
import pytest

from fluidisim_b200 import scenes
from fluidisim_b200.batch import project_batch
from fluidisim_b200.delta3d import Volume3

pytestmark = pytest.mark.gpu

SCALE, K1 = -1025.0 * 60.0, 1.0 / (1025.0 * 60.0)


def volume(shape, multigrid, seed=5):
    nx, ny, nz = shape
    dx = 0.1
    i, j = np.meshgrid(np.arange(nx), np.arange(ny), indexing="xy")
    v = Volume3.configure(nx, ny, nz, dx, 1025.0, 9.81)
    if multigrid:
        v.enable_multigrid()
    rest = float(np.float32(0.55 * nz * dx))
    v.set_free_surface((rest + 0.05 * nz * dx * np.sin(7.0 * i / nx + 3.0 * j / ny + seed)).astype(np.float32).ravel(), rest)
    rng = scenes.SplitMix64(seed)
    return v, [rng.uniform_array(n, -1.0, 1.0) for n in scenes.face_counts(nx, ny, nz)]


def restart(volumes):
    for v, velocity in volumes:
        v.set_velocity(*velocity)
        v.reset_pressure()


def batch(volumes, workers):
    n = len(volumes)
    restart(volumes)
    t = time.perf_counter()
    reports, statuses = project_batch([v for v, _ in volumes], [SCALE] * n, [K1] * n, threads=workers)
    t = time.perf_counter() - t
    assert statuses == [0] * n
    return t, reports


@pytest.mark.parametrize("shape,multigrid", [((40, 40, 40), True), ((45, 33, 27), False), ((75, 61, 17), False)])
def test_a_batch_runs_side_by_side(shape, multigrid):
    volumes = [volume(shape, multigrid, 5 + q) for q in range(8)]
    one = min(batch(volumes, 1)[0] for _ in range(5))
    many = min(batch(volumes, 8)[0] for _ in range(5))
    for v, _ in volumes:
        v.close()
    share = 0.8 if shape == (75, 61, 17) else 0.53  # 77,775 cells, two per thread on every SM: half of the SMs each
    assert many < share * one, (many, one)


@pytest.mark.parametrize("shape,multigrid", [((48, 48, 48), True), ((61, 35, 31), False)])
def test_two_threads_run_side_by_side(shape, multigrid):
    volumes = [volume(shape, multigrid, 5 + q) for q in range(2)]

    def work(v, velocity):
        for _ in range(10):
            v.set_velocity(*velocity)
            v.reset_pressure()
            v.project_mobile3(SCALE, K1)

    def both(threads):
        pool = [threading.Thread(target=work, args=x) for x in volumes]
        t = time.perf_counter()
        for p in pool:
            p.start()
            if not threads:
                p.join()
        for p in pool:
            p.join()
        return time.perf_counter() - t

    one = min(both(False) for _ in range(5))
    two = min(both(True) for _ in range(5))
    for v, _ in volumes:
        v.close()
    assert two < 0.8 * one, (two, one)


@pytest.mark.parametrize("workers", [2, 3, 5, 20])
def test_the_result_does_not_depend_on_the_share(workers):
    """Every way a grid is cut down: parts of sums over 64 and below, chunks of a narrow and of a high volume, CTAs that
    stand in for two and for four, with and without a remainder, and one cell to a thread and two."""
    shapes = [((16, 16, 16), True), ((64, 64, 64), True), ((34, 10, 22), True), ((2, 2, 1000), True), ((16, 16, 480), True),
              ((130, 36, 12), True), ((9, 8, 7), False), ((45, 33, 27), False), ((31, 33, 37), False), ((75, 61, 17), False),
              ((101, 67, 22), False)]
    alone = []
    for s, mg in shapes:
        v, velocity = volume(s, mg)
        v.set_velocity(*velocity)
        alone.append((v.project_mobile3(SCALE, K1, 40), v.pressure()))
        v.close()
    volumes = [volume(s, mg) for s, mg in shapes]
    restart(volumes)
    n = len(volumes)
    reports, statuses = project_batch([v for v, _ in volumes], [SCALE] * n, [K1] * n, max_iters=40, threads=workers)
    assert statuses == [0] * n
    for (v, _), r, (ra, p) in zip(volumes, reports, alone):
        assert r == ra and np.array_equal(v.pressure(), p)
        v.close()
