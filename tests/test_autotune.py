"""The autotuner of the per-patch path times its candidates as they will run: several volumes at once (no GPU: the volumes
and the batch are stand-ins)."""
import time

from fluidisim_b200 import batch


def test_a_candidate_that_is_fast_alone_and_slow_together_is_not_kept(monkeypatch):
    class Stand:
        def __init__(self, kernels):
            self.kernels = kernels

        def set_velocity(self, *a):
            pass

        def reset_pressure(self):
            pass

        def project_mobile3(self, *a):
            time.sleep({0: 0.004, 1: 0.002, 2: 0.008}[self.kernels])

        def close(self):
            pass

    def together(vols, scales, k1s, threads=0):
        time.sleep({0: 0.004, 1: 0.016, 2: 0.032}[vols[0].kernels])
        return [None] * len(vols), [0] * len(vols)

    monkeypatch.setattr(batch, "configure", lambda scene, kernels=0, levels=0: Stand(kernels))
    monkeypatch.setattr(batch, "project_batch", together)
    scene = dict(nx=24, ny=16, nz=16, u=None, v=None, w=None, rho=1025.0, dt=1.0 / 60.0)
    tuned = batch.autotune({"small": [scene]}, repeats=2)
    assert tuned["small"].kernels == 0
