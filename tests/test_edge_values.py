"""Fields with infinities and NaN on their outermost nodes (GPU): a set that reads the ring slots because it is small gives
what it gives as part of a set that reads window pairs, bit for bit, for particles in the edge cells and stages beyond."""
import numpy as np
import pytest

from pygranite_b200 import capi

pytestmark = pytest.mark.gpu

WINDOWS, PER_WINDOW, FEW = 3, 10, 900


@pytest.mark.parametrize("storage", [0, 1, 2])
@pytest.mark.parametrize("rk4", [0, 1])
@pytest.mark.parametrize("shape", [(7, 9, 11), (1, 6, 8), (13, 15)])
def test_small_sets_clamp_like_pairs(shape, rk4, storage):
    dim = len(shape)
    rng = np.random.default_rng(100 * storage + 10 * rk4 + dim)
    wind = []
    for _ in range(WINDOWS + 1):
        planes = []
        for _ in range(dim):
            p = (rng.standard_normal(shape) * 0.3).astype(np.float32)
            edge = np.ones(shape, bool)
            edge[tuple(slice(1, -1) if s > 2 else slice(None) for s in shape)] = False
            bad = edge & (rng.random(shape) < 0.3)
            p[bad] = rng.choice(np.array([np.inf, -np.inf, np.nan], np.float32), int(bad.sum()))
            planes.append(p)
        wind.append(planes)
    few = np.concatenate([rng.uniform(-0.3, np.array(shape[::-1]) + 0.3, (FEW // 2, dim)),
                          rng.uniform(0.0, np.array(shape[::-1]), (FEW // 2, dim))]).astype(np.float32)
    many = np.concatenate([few, rng.uniform(0, shape[::-1], (300_000, dim)).astype(np.float32)])
    settings = dict(Space=0 if dim == 3 else 1, Integrator=rk4, WindfieldMode=1, DeltaT=0.5, GridScale=[1.0] * dim,
                    Offset=[0.0] * dim, DataTimeDistance=0.5 * PER_WINDOW, SaveInterval=5,
                    MaximumSimulationTime=0.5 * PER_WINDOW * WINDOWS)
    got = []
    for seeds, launches in ((few, 1), (many, WINDOWS)):
        e = capi.Engine(capi.settings_from_reference(settings, ring_slots=WINDOWS + 1, storage=storage))
        e.set_seeds(seeds)
        for k, planes in enumerate(wind):
            e.load_windfield(k, planes)
        e.run(lambda k: 1 if k <= WINDOWS else 0)
        assert e.stats().launches == launches      # ring slots, pairs
        r = e.results()
        got.append((r["trajectories"][:FEW], r["status"][:FEW]))
        e.close()
    assert np.array_equal(got[0][1], got[1][1])
    assert np.array_equal(got[0][0], got[1][0], equal_nan=True)
    assert not np.isfinite(got[0][0]).all()        # the edge was reached
    assert (got[0][1] == 0).any()
