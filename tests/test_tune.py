"""The autotuner keeps the settings of an engine whose automatic choices are the fastest (GPU)."""
import numpy as np
import pytest

from pygranite_b200 import capi

pytestmark = pytest.mark.gpu


def test_few_particles_keep_their_automatic_blocks():
    """1,000 particles run in blocks of 4 threads untuned, where blocks of 64 take a third longer."""
    shape, n, windows = (16, 24, 24), 1000, 10
    rng = np.random.default_rng(3)
    e = capi.Engine(capi.settings_from_reference(
        dict(Space=0, Integrator=1, WindfieldMode=1, DeltaT=1.0, DataTimeDistance=10.0, GridScale=[1.0] * 3, Offset=[0.0] * 3,
             SaveInterval=0, MaximumSimulationTime=10.0 * windows), ring_slots=windows + 1))
    e.set_seeds((rng.uniform(0.3, 0.7, (n, 3)) * shape[::-1]).astype(np.float32))
    for k in range(windows + 1):
        e.load_windfield(k, [(rng.standard_normal(shape) * 0.3).astype(np.float32) for _ in range(3)])
    before = bytes(e.settings())
    e.run(lambda k: 1 if k <= windows else 0)
    ref = e.final_positions()
    r = e.tune(trial_steps=100)
    assert r.kept == 1 and r.trials >= 2 and r.particle_steps_per_s > 0
    assert bytes(e.settings()) == before
    e.run(lambda k: 1 if k <= windows else 0)
    assert np.array_equal(e.final_positions(), ref)
    e.close()


def test_settings_that_lose_are_replaced():
    """One thread a block is the slowest way to run 60,000 particles."""
    shape, n, windows = (16, 24, 24), 60_000, 10
    rng = np.random.default_rng(4)
    e = capi.Engine(capi.settings_from_reference(
        dict(Space=0, Integrator=1, WindfieldMode=1, DeltaT=1.0, DataTimeDistance=10.0, GridScale=[1.0] * 3, Offset=[0.0] * 3,
             SaveInterval=0, MaximumSimulationTime=10.0 * windows), ring_slots=windows + 1, block_size=1))
    e.set_seeds((rng.uniform(0.3, 0.7, (n, 3)) * shape[::-1]).astype(np.float32))
    for k in range(windows + 1):
        e.load_windfield(k, [(rng.standard_normal(shape) * 0.3).astype(np.float32) for _ in range(3)])
    r = e.tune(trial_steps=100)
    s = e.settings()
    assert r.kept == 0
    assert (s.layout, s.block_size, s.sort_interval, s.grid_waves) == (r.layout, r.block_size, r.sort_interval, r.grid_waves)
    assert s.block_size >= 64
    e.close()
