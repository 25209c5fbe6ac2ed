"""Deferred values of dynamic volumes where the ring is reused (GPU): a particle that stops between two records keeps
the values of its last step, whose snapshots must still be in the ring when they are evaluated."""
import numpy as np
import pytest

from tests import harness as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,n,per_window,save", [((40, 50, 60), 700, 10, 4), ((12, 20, 24), 9000, 40, 8),
                                                     ((30, 40), 5000, 128, 64)])
def test_stopped_particles_keep_their_last_values(shape, n, per_window, save):
    rng = np.random.default_rng(n + per_window)
    dim, windows = len(shape), 5
    wind = [[(rng.standard_normal(shape) * 0.5).astype(np.float32) for _ in range(dim)] for _ in range(windows + 1)]
    seeds = rng.uniform(0, shape[::-1], (n, dim)).astype(np.float32)
    volumes = [{"t": rng.standard_normal(shape).astype(np.float32)} for _ in wind]
    settings = dict(Space=0 if dim == 3 else 1, Integrator=1, WindfieldMode=1, DeltaT=0.25, SaveInterval=save,
                    DataTimeDistance=0.25 * per_window, GridScale=[1.0] * dim, Offset=[0.0] * dim,
                    MaximumSimulationTime=0.25 * (per_window * windows - 1), AdditionalVolumeMode=2,
                    AdditionalCompute=["t + x*u", "v - y"])
    eng = H.run_engine(settings, wind, seeds, volumes=volumes)
    ref = H.run_oracle(settings, wind, seeds, volumes=volumes, precision="f32")
    H.assert_same(eng, ref)
    assert np.array_equal(eng["volume_info"]["t"], ref["volume_info"]["t"])
    for k in range(2):
        assert np.array_equal(eng["compute_info"][k], ref["compute_info"][k])
