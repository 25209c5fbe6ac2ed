"""Blocks of less than a warp (GPU): counts around the lines of the automatic choice and block sizes given by the
settings, bit for bit against the float32 oracle; every particle-step is counted."""
import numpy as np
import pytest

from pygranite_b200 import capi
from tests import harness as H

pytestmark = pytest.mark.gpu


def problem(shape, n):
    rng = np.random.default_rng(n)
    dim = len(shape)
    wind = [[(rng.standard_normal(shape) * 0.3).astype(np.float32) for _ in range(dim)] for _ in range(3)]
    seeds = rng.uniform(0, shape[::-1], (n, dim)).astype(np.float32)
    settings = dict(Space=0 if dim == 3 else 1, Integrator=1, WindfieldMode=1, DeltaT=0.5, SaveInterval=3,
                    DataTimeDistance=4.0, GridScale=[1.0] * dim, Offset=[0.0] * dim, MaximumSimulationTime=8.0)
    return settings, wind, seeds


@pytest.mark.parametrize("shape", [(6, 9, 11), (14, 13)])
@pytest.mark.parametrize("n,block", [(1, 0), (5, 0), (2367, 0), (2369, 0), (10_657, 0), (21_313, 0), (700, 1), (700, 5),
                                     (700, 33)])
def test_partial_warps_equal_the_oracle(shape, n, block):
    settings, wind, seeds = problem(shape, n)
    ref = H.run_oracle(settings, wind, seeds, precision="f32")
    e = capi.Engine(capi.settings_from_reference(settings, ring_slots=3, block_size=block))
    e.set_seeds(seeds)
    for k, s in enumerate(wind):
        e.load_windfield(k, s)
    e.run(lambda k: 1 if k < len(wind) else 0)
    H.assert_same(e.results(), ref)
    assert e.info().particle_steps == ref["particle_steps"]
    e.close()


def test_alive_counts_need_whole_warps():
    settings, wind, seeds = problem((6, 9, 11), 900)
    settings.update(MinimumAliveParticles=600)
    ref = H.run_oracle(settings, wind, seeds, precision="f32")
    H.assert_same(H.run_engine(settings, wind, seeds), ref)
