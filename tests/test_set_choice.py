"""Which of the two ways a set with volumes and records goes (GPU): ring slots, one launch for all resident windows, where
few particles share the grid; pairs, a launch a window, where the evaluation in the step kernel would cost more."""
import numpy as np
import pytest

from pygranite_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,n,pairs", [((16, 24, 24), 6_000, False), ((16, 24, 24), 20_000, True),
                                           ((16, 24, 24), 40_000, True), ((40, 130, 130), 25_000, False),
                                           ((40, 130, 130), 60_000, True)])
def test_plain_runs(shape, n, pairs):
    windows = 5
    assert launches(shape, n, windows) == (windows if pairs else 1)


def test_ring_slots_asked_for_stay_in_one_launch():
    """With the layout given there are no pairs to go back to."""
    assert launches((16, 24, 24), 20_000, 5, layout=1) == 1


def launches(shape, n, windows, per_window=10, **kw):
    rng = np.random.default_rng(n)
    e = capi.Engine(capi.settings_from_reference(
        dict(Space=0, Integrator=1, WindfieldMode=1, AdditionalVolumeMode=1, DeltaT=1.0, GridScale=[1.0] * 3, CurvatureMode=1,
             Offset=[0.0] * 3, DataTimeDistance=float(per_window), SaveInterval=per_window,
             MaximumSimulationTime=float(windows * per_window)), ring_slots=windows + 1, **kw))
    e.set_seeds((rng.uniform(0.3, 0.7, (n, 3)) * shape[::-1]).astype(np.float32))
    plane = (rng.standard_normal(shape) * 0.05).astype(np.float32)
    for k in range(windows + 1):
        e.load_windfield(k, [plane] * 3)
    e.load_volume(0, 0, plane)
    e.run(lambda k: 1 if k <= windows else 0)
    count = e.stats().launches
    e.close()
    return count
