"""Sets on either side of the choice between window pairs and ring slots, against the float32 oracle (GPU).

The choice depends on particles, nodes and steps a window, and with it launches span one window or many, and volumes
and expressions are evaluated in the step kernel or after it.  Every value stays the same bit for bit."""
import numpy as np
import pytest

from tests import harness as H

pytestmark = pytest.mark.gpu

# (shape, particles, steps a window, record every, expressions): ring slots in the first four, pairs in the rest
CASES = [((40, 50, 60), 700, 10, 4, True), ((24, 100, 90), 20_000, 6, 0, False), ((90, 120), 3000, 10, 3, True),
         ((200, 210), 70_000, 10, 7, False), ((12, 20, 24), 9000, 40, 8, True), ((8, 9, 10), 150_000, 10, 10, False),
         ((30, 40), 5000, 128, 64, True)]


@pytest.mark.parametrize("shape,n,per_window,save,extras", CASES, ids=lambda v: str(v).replace(" ", ""))
@pytest.mark.parametrize("ring", [0, 6])
def test_small_sets_equal_the_oracle(shape, n, per_window, save, extras, ring):
    rng = np.random.default_rng(n + per_window)
    dim, windows = len(shape), 5
    wind = [[(rng.standard_normal(shape) * 0.5).astype(np.float32) for _ in range(dim)] for _ in range(windows + 1)]
    seeds = rng.uniform(0, shape[::-1], (n, dim)).astype(np.float32)
    settings = dict(Space=0 if dim == 3 else 1, Integrator=1, WindfieldMode=1, DeltaT=0.25, SaveInterval=save,
                    DataTimeDistance=0.25 * per_window, GridScale=[1.0] * dim, Offset=[0.0] * dim,
                    MaximumSimulationTime=0.25 * (per_window * windows - 1), CurvatureMode=1 if dim == 3 else 0)
    volumes = None
    if extras:
        volumes = [{"t": rng.standard_normal(shape).astype(np.float32)} for _ in wind]
        settings.update(AdditionalVolumeMode=2, AdditionalCompute=["t + x*u", "v - y"])
    eng = H.run_engine(settings, wind, seeds, volumes=volumes, RingSlots=ring)
    ref = H.run_oracle(settings, wind, seeds, volumes=volumes, precision="f32")
    H.assert_same(eng, ref, ("trajectories", "status") + (("total_curvature",) if dim == 3 else ()))
    if extras:
        assert np.array_equal(eng["volume_info"]["t"], ref["volume_info"]["t"])
        for k in range(2):
            assert np.array_equal(eng["compute_info"][k], ref["compute_info"][k])
