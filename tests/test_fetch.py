"""Results to host memory (GPU): tiles and chunks of every shape give the oracle's rows, in pageable and page-locked
arrays, with records of particles that retired on the way."""
import numpy as np
import pytest

from pygranite_b200 import capi
from tests import harness as H

pytestmark = pytest.mark.gpu


def problem(shape, n, steps, save):
    rng = np.random.default_rng(n + steps)
    dim = len(shape)
    wind = [[(rng.standard_normal(shape) * 0.4).astype(np.float32) for _ in range(dim)] for _ in range(3)]
    seeds = rng.uniform(0, shape[::-1], (n, dim)).astype(np.float32)
    settings = dict(Space=0 if dim == 3 else 1, Integrator=0, WindfieldMode=1, DeltaT=0.5, SaveInterval=save,
                    DataTimeDistance=0.25 * steps, GridScale=[1.0] * dim, Offset=[0.0] * dim,
                    MaximumSimulationTime=0.5 * steps, AbortMode=2, MaximumLength=3.0)
    return settings, wind, seeds


def engine(settings, wind, seeds, **extra):
    e = capi.Engine(capi.settings_from_reference(settings, ring_slots=3, **extra))
    e.set_seeds(seeds)
    for k, s in enumerate(wind):
        e.load_windfield(k, s)
    e.run(lambda k: 1 if k < len(wind) else 0)
    return e


@pytest.mark.parametrize("shape", [(5, 6, 7), (9, 8)])
@pytest.mark.parametrize("n,steps,save", [(1, 8, 0), (127, 8, 8), (129, 16, 2), (1025, 16, 2), (33, 64, 1), (1023, 66, 1)])
def test_rows_equal_the_oracle(shape, n, steps, save):
    settings, wind, seeds = problem(shape, n, steps, save)
    ref = H.run_oracle(settings, wind, seeds, precision="f32")
    e = engine(settings, wind, seeds, sort_interval=1, steps_per_launch=3)
    for pinned in (False, True):
        H.assert_same(e.results(pinned=pinned), ref, ("trajectories", "status", "lengths"))
    assert np.array_equal(e.final_positions(), ref["trajectories"][:, -1])
    e.close()


def test_chunks_of_large_results():
    """Rows of 31 records, over 32 MB in all and not a whole number of chunks."""
    settings, wind, seeds = problem((5, 6, 7), 250_007, 60, 2)
    ref = H.run_oracle(settings, wind, seeds, precision="f32")
    e = engine(settings, wind, seeds)
    for pinned in (False, True):
        H.assert_same(e.results(pinned=pinned), ref, ("trajectories", "status", "lengths"))
    e.close()
