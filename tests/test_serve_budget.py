"""The limit on the request server's field in device memory (GPU): nothing of it beyond the ring at 0, the packed field
with one pair, the field with all pairs.  Results are the float32 oracle's in each, and the device memory held stays
within the limit and what a server with limit 0 holds."""
import ctypes
import gc

import numpy as np
import pytest

from oracle import oracle as orc
from pygranite_b200 import capi

pytestmark = pytest.mark.gpu

SNAPSHOTS, SHAPE = 12, (40, 60, 70)
SLOT = 40 * 60 * 70 * 3 * 4                      # float32, planar
PAIR = 43 * 63 * 73 * 8 * 4
LIMITS = {"host": 0, "one byte short": SNAPSHOTS * SLOT + PAIR - 1, "one pair": SNAPSHOTS * SLOT + PAIR + 1024 * SNAPSHOTS,
          "all pairs": SNAPSHOTS * (SLOT + PAIR + 1024)}


def used():
    a, b = ctypes.c_int64(0), ctypes.c_int64(0)
    assert capi.lib().gr_device_cache_stats_get(0, ctypes.byref(a), ctypes.byref(b)) == 0
    return b.value


@pytest.fixture(scope="module")
def problem():
    rng = np.random.default_rng(8)
    wind = [[(rng.standard_normal(SHAPE) * 0.5).astype(np.float32) for _ in range(3)] for _ in range(SNAPSHOTS)]
    base = dict(Space=0, Integrator=1, WindfieldMode=1, DeltaT=0.25, DataTimeDistance=1.0, GridScale=[1.0] * 3,
                Offset=[0.0] * 3, SaveInterval=0, MaximumSimulationTime=SNAPSHOTS - 1.0)
    reqs = [dict(seeds=rng.uniform(0, SHAPE[::-1], (n, 3)).astype(np.float32), k0=k0, steps=m)
            for n, k0, m in [(700, 0, 44), (33, 9, 20), (1025, 30, 14)]]
    for r in reqs:
        ref = orc.run(orc.settings(**base), orc.Inputs(wind=wind, seeds=r["seeds"]), precision="f32", start_step=r["k0"],
                      step_limit=r["k0"] + r["steps"])
        r["ref"] = ref["status"], ref["trajectories"][:, -1]
    return base, wind, reqs


def serve(problem, limit):
    """Device bytes of the server, bytes copied to the device by two rounds of requests."""
    base, wind, reqs = problem
    gc.collect()          # what earlier tests left is not to be given back in between
    before = used()
    srv = capi.Server(capi.settings_from_reference(base), SNAPSHOTS, SHAPE, hbm_budget=4 << 20, field_budget=limit)
    held = used() - before
    for k, s in enumerate(wind):
        srv.set_snapshot(k, s)
    srv.start()
    for again in range(2):
        ids = [srv.submit(r["seeds"], 0.25 * r["k0"], r["steps"], 1) for r in reqs]
        for rid, r in zip(ids, reqs):
            assert srv.wait(rid, 60.0) == capi.GR_REQ_DONE
            pos, st, _ = srv.result(rid)
            srv.release(rid)
            assert np.array_equal(st, r["ref"][0]) and np.array_equal(pos, r["ref"][1])
    moved = srv.stats().h2d_bytes
    srv.close()
    return held, moved


@pytest.mark.parametrize("name", list(LIMITS))
def test_the_field_keeps_its_limit(problem, name):
    ring, streamed = serve(problem, 0)
    held, moved = serve(problem, LIMITS[name])
    assert held <= ring - 4 * SLOT - PAIR + max(LIMITS[name], 4 * SLOT + PAIR) + (64 << 10)
    assert (moved == streamed) == (name in ("host", "one byte short"))
    if name == "all pairs":
        assert held > SNAPSHOTS * SLOT + (SNAPSHOTS - 1) * PAIR


def test_without_a_limit_the_field_stays_on_the_device(problem):
    assert serve(problem, -1)[1] < SLOT
