"""Admission staging of the request server (GPU): as large as the requests at hand, from the library's host cache, and grown
by larger ones; results stay those of the float32 oracle."""
import ctypes
import gc

import numpy as np
import pytest

from oracle import oracle as orc
from pygranite_b200 import capi

pytestmark = pytest.mark.gpu


def cache():
    st = capi.HostCacheStats()
    assert capi.lib().gr_host_cache_stats_get(ctypes.byref(st)) == 0
    return st


@pytest.mark.parametrize("dim", [2, 3])
def test_staging_grows_with_the_requests(dim):
    shape = (24, 20) if dim == 2 else (8, 9, 10)
    rng = np.random.default_rng(dim)
    wind = [[(rng.standard_normal(shape) * 0.2).astype(np.float32) for _ in range(dim)] for _ in range(3)]
    base = dict(Space=0 if dim == 3 else 1, Integrator=1, WindfieldMode=1, DeltaT=0.5, DataTimeDistance=2.0,
                GridScale=[1.0] * dim, Offset=[0.0] * dim, SaveInterval=0, MaximumSimulationTime=4.0)
    srv = capi.Server(capi.settings_from_reference(base), 3, shape, hbm_budget=100 << 20)
    for k, s in enumerate(wind):
        srv.set_snapshot(k, s)
    srv.start()
    gc.collect()          # what earlier tests left is not to be given back in between
    live, made, held = cache().live_bytes, cache().allocations + cache().reuses, []
    for n in (1, 87_382, 104_857, 104_858, 350_000, 7):     # around 2 MB and 8 MB blocks
        seeds = rng.uniform(0, shape[::-1], (n, dim)).astype(np.float32)
        for rk4 in (1, 0):
            rid = srv.submit(seeds, 0.0, 8, rk4)
            assert srv.wait(rid, 60.0) == capi.GR_REQ_DONE
            pos, st, _ = srv.result(rid)
            srv.release(rid)
            some = slice(None) if n < 10_000 else slice(None, None, 50)
            ref = orc.run(orc.settings(**dict(base, Integrator=rk4)), orc.Inputs(wind=wind, seeds=seeds[some]),
                          precision="f32")
            assert np.array_equal(st[some], ref["status"])
            assert np.array_equal(pos[some], ref["trajectories"][:, -1])
        held.append(cache().live_bytes - live)
    assert held[0] == 2 * (2 << 20)                         # two staging buffers
    assert held[-1] == held[-2] and held[-2] <= 2 * (32 << 20)
    assert cache().allocations + cache().reuses - made <= 6
    srv.close()
    assert cache().live_bytes == live
