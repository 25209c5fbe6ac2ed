"""Runs large enough for the automatic sort of the seeds, bit for bit against the float32 oracle (GPU).

The order of the particles changes nothing; particles whose lifetime is zero retire in that first pass."""
import numpy as np
import pytest

from pygranite_b200 import capi
from tests import harness as H

pytestmark = pytest.mark.gpu


def problem(shape, n, windows=4):
    rng = np.random.default_rng(n)
    dim = len(shape)
    wind = [[(rng.standard_normal(shape) * 0.4).astype(np.float32) for _ in range(dim)] for _ in range(windows + 1)]
    seeds = rng.uniform(0, shape[::-1], (n, dim)).astype(np.float32)
    settings = dict(Space=0 if dim == 3 else 1, Integrator=1, WindfieldMode=1, DeltaT=0.5, DataTimeDistance=16.0,
                    GridScale=[1.0] * dim, Offset=[0.0] * dim, SaveInterval=16, MaximumSimulationTime=16.0 * windows)
    return settings, wind, seeds


@pytest.mark.parametrize("shape,n", [((12, 20, 24), 65536), ((12, 20, 24), 131071), ((65, 70), 200003)])
def test_sorted_seeds_equal_the_oracle(shape, n):
    settings, wind, seeds = problem(shape, n)
    volumes = [{"t": np.random.default_rng(5).standard_normal(shape).astype(np.float32)}]
    settings.update(AdditionalVolumeMode=1, AdditionalCompute=["t + x*u"], CurvatureMode=1 if len(shape) == 3 else 0)
    eng = H.run_engine(settings, wind, seeds, volumes=volumes)
    ref = H.run_oracle(settings, wind, seeds, volumes=volumes, precision="f32")
    H.assert_same(eng, ref, ("trajectories", "status") + (("total_curvature",) if len(shape) == 3 else ()))
    assert np.array_equal(eng["volume_info"]["t"], ref["volume_info"]["t"])
    assert np.array_equal(eng["compute_info"][0], ref["compute_info"][0])


def test_lifetimes_of_zero_retire_before_the_first_step():
    settings, wind, seeds = problem((12, 20, 24), 100_001)
    life = np.random.default_rng(6).integers(0, 3, len(seeds)).astype(np.int32) * 64
    eng = capi.Engine(capi.settings_from_reference(settings, ring_slots=len(wind)))
    eng.set_seeds(seeds)
    eng.set_lifetimes(life)
    for k, s in enumerate(wind):
        eng.load_windfield(k, s)
    eng.run(lambda k: 1 if k < len(wind) else 0)
    out = eng.results()
    eng.close()
    still = life == 0
    assert np.array_equal(out["trajectories"][still], np.repeat(seeds[still][:, None], out["info"].records, axis=1))
    assert not out["status"][still].any()
    whole = H.run_oracle(settings, wind, seeds, precision="f32")
    for k in (64, 128):
        cut = H.run_oracle(dict(settings, MaximumSimulationTime=0.5 * k), wind, seeds, precision="f32")
        mine = life == k
        m = cut["trajectories"].shape[1]
        assert np.array_equal(out["trajectories"][mine, :m], cut["trajectories"][mine])
        assert np.array_equal(out["status"][mine], cut["status"][mine])
    assert whole["trajectories"].shape[1] == out["info"].records
