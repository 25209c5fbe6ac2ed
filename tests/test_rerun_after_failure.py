"""A run that follows a failed one on the same engine (GPU).  The failed run returns while its launches and passes are
still queued, among them the copy of a live count; the next run may not take that count for its own."""
import time

import numpy as np
import pytest

from pygranite_b200 import capi

pytestmark = pytest.mark.gpu

SHAPE, N, PER_WINDOW = (8, 8, 1000), 200_000, 600


def test_live_counts_of_a_failed_run():
    """Particles below y = 4 leave the domain in the first window, those above stay; runs of the first kind fail after
    their last window, runs of the second kind start at every moment of the queue that they left."""
    rng = np.random.default_rng(5)
    u = np.full(SHAPE, 0.05, np.float32)
    u[:, :4] = 2.0
    wind = [u, np.full(SHAPE, 1e-4, np.float32), np.full(SHAPE, 1e-4, np.float32)]

    def seeds(lo, hi):
        return np.stack([rng.uniform(5, 9, N), rng.uniform(lo, hi, N), rng.uniform(1, 6, N)], axis=1).astype(np.float32)

    leaving, staying = seeds(1, 3), seeds(5, 6.5)
    st = capi.settings_from_reference(dict(Space=0, Integrator=1, WindfieldMode=1, DeltaT=1.0, CurvatureMode=0,
                                           DataTimeDistance=float(PER_WINDOW), GridScale=[1.0] * 3, Offset=[0.0] * 3,
                                           SaveInterval=0, MaximumSimulationTime=2.0 * PER_WINDOW),
                                      ring_slots=4, sort_interval=1)

    def engine():
        e = capi.Engine(st)
        e.set_seeds(staying)
        for k in range(3):
            e.load_windfield(k, wind)
        return e

    e = engine()
    e.run(lambda k: 1 if k < 3 else 0)
    ref = e.final_positions()
    took = e.stats().run_ms
    e.close()
    e = engine()
    for delay in np.linspace(0.0, 1.2 * took, 240):
        e.set_seeds(leaving)
        with pytest.raises(capi.GraniteError):
            e.run(lambda k: -1 if k == 3 else 1)
        until = time.perf_counter() + 1e-3 * delay
        e.set_seeds(staying)
        while time.perf_counter() < until:
            pass
        e.run(lambda k: 1 if k < 3 else 0)
        assert np.array_equal(e.final_positions(), ref), f"{delay:.2f} ms after the failed run"
    e.close()
