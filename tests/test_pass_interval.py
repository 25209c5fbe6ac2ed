"""Automatic compaction passes come every so many windows, however many launches a window takes (GPU)."""
import numpy as np
import pytest

from pygranite_b200 import capi

pytestmark = pytest.mark.gpu


def other_launches(save, windows=20, per_window=10, steps_per_launch=0, **more):
    """Launches beside the steps, the records' deferred evaluations taken off."""
    shape, n = (16, 24, 24), 100_000
    rng = np.random.default_rng(1)
    e = capi.Engine(capi.settings_from_reference(
        dict(Space=0, Integrator=1, WindfieldMode=1, AdditionalVolumeMode=1, DeltaT=1.0, GridScale=[1.0] * 3, Offset=[0.0] * 3,
             DataTimeDistance=float(per_window), SaveInterval=save, MaximumSimulationTime=float(windows * per_window), **more),
        ring_slots=windows + 1, steps_per_launch=steps_per_launch))
    e.set_seeds((rng.uniform(0.4, 0.6, (n, 3)) * shape[::-1]).astype(np.float32))
    for k in range(windows + 1):
        e.load_windfield(k, [(rng.standard_normal(shape) * 0.05).astype(np.float32) for _ in range(3)])
    e.load_volume(0, 0, rng.standard_normal(shape).astype(np.float32))
    e.run(lambda k: 1 if k <= windows else 0)
    st, records = e.stats(), e.info().records
    e.close()
    return st.aux_launches - records, st.launches


def test_records_do_not_add_passes():
    base, launches = other_launches(10)
    every, more = other_launches(1)
    assert launches == 20 and more == 200      # deferred: a launch ends at every record
    assert every == base


def test_short_launches_do_not_add_passes():
    base, _ = other_launches(0)
    short, more = other_launches(0, steps_per_launch=3)
    assert more >= 67
    assert short == base


def test_length_aborts_are_retired_every_8_windows():
    base, _ = other_launches(0, CurvatureMode=3)
    ends, _ = other_launches(0, CurvatureMode=3, AbortMode=2, MaximumLength=1e9)
    assert ends == base + 3        # after 8 and 16 windows instead of after 16: a pass is three launches
