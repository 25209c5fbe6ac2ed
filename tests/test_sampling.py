"""Sampling from window pairs and straight from ring slots, bit for bit against the float32 oracle (GPU).

Both wind layouts share the sample cache; the ring layout clamps corner indices into the grid and zeroes the 3D
corners outside, so the cases sit at the edges: axes of one and two nodes, particles on and beside every face, cells
that change at every step, particle counts around a warp and a block, 16-bit storage.
"""
import numpy as np
import pytest

from oracle import oracle as orc
from pygranite_b200 import workloads as W
from tests import harness as H

pytestmark = pytest.mark.gpu

STORES = {"f32": "Float32", "bf16": "BFloat16", "f16": "Float16"}
# (shape, particles, per-step displacement in cells): one- and two-node axes, ragged counts, fast and slow particles
GRIDS = [((1, 5, 6), 33, 0.3), ((2, 2, 2), 129, 0.2), ((7, 1, 9), 31, 0.6), ((9, 13, 11), 2049, 1.7),
         ((16, 24, 20), 4097, 0.05), ((1, 7), 65, 0.3), ((2, 2), 1, 0.1), ((33, 17), 2047, 0.9), ((24, 40), 4100, 0.04)]


def problem(shape, n, speed, seed, windows=4):
    """Random fields, seeds over the whole domain and a cell's breadth around every face."""
    rng = np.random.default_rng(seed)
    dim = len(shape)
    wind = [[(rng.standard_normal(shape) * speed).astype(np.float32) for _ in range(dim)] for _ in range(windows + 1)]
    hi = np.array(shape[::-1], np.float64)
    seeds = rng.uniform(0, hi, (n, dim))
    face = rng.integers(0, 2 * dim, n)
    near = rng.random(n) < 0.5
    for d in range(dim):
        for side in (0, 1):
            pick = near & (face == 2 * d + side)
            seeds[pick, d] = (hi[d] if side else 0.0) + rng.uniform(-0.6, 0.6, int(pick.sum()))
    settings = dict(Space=0 if dim == 3 else 1, Integrator=1, WindfieldMode=1, DeltaT=1.0, DataTimeDistance=4.0,
                    GridScale=[1.0] * dim, Offset=[0.0] * dim, SaveInterval=1, MaximumSimulationTime=4.0 * windows)
    return settings, wind, seeds.astype(np.float32)


@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("store", sorted(STORES))
@pytest.mark.parametrize("shape,n,speed", GRIDS, ids=lambda v: str(v).replace(" ", ""))
def test_sampling_equals_the_oracle(shape, n, speed, store, layout):
    import pygranite_b200 as pg
    settings, wind, seeds = problem(shape, n, speed, seed=n + layout)
    stored = [[W.round_storage(p, store) for p in s] for s in wind]
    options = [dict(), dict(Integrator=0), dict(WindfieldMode=0), dict(ReferenceFilter=True)]
    options += [dict(CurvatureMode=1)] if len(shape) == 3 else [dict(BorderMode=1), dict(BorderMode=3)]
    for opt in options:
        opt = dict(opt)
        extra = dict(WindStorage=getattr(pg.WindStorage, STORES[store]), WindLayout=layout)
        if opt.pop("ReferenceFilter", False):
            extra["ReferenceFilter"] = True
        s = dict(settings, **opt)
        eng = H.run_engine(s, wind, seeds, **extra)
        ref = orc.run(orc.settings(**s), orc.Inputs(wind=stored, seeds=seeds), "f32",
                      filter_weights=int("ReferenceFilter" in extra))
        H.assert_same(eng, ref, ("trajectories", "status") + (("total_curvature",) if "CurvatureMode" in opt else ()))
