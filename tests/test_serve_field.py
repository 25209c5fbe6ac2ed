"""Where the request server keeps its field (GPU): on the device, or in host memory behind a 4-slot ring.  Requests that
span sweeps, windows and both integrators give the float32 oracle's results either way."""
import numpy as np
import pytest

from oracle import oracle as orc
from pygranite_b200 import capi
from pygranite_b200 import workloads as W

pytestmark = pytest.mark.gpu

SNAPSHOTS = 8


@pytest.mark.parametrize("resident", ["1", "0"])
@pytest.mark.parametrize("shape,storage", [((5, 9, 11), 0), ((12, 20, 24), 1), ((30, 41), 0), ((32, 48), 2)])
def test_requests_equal_the_oracle(shape, storage, resident, monkeypatch):
    monkeypatch.setenv("GR_SERVE_RESIDENT", resident)
    rng = np.random.default_rng(storage + len(shape))
    dim = len(shape)
    snaps = [[(rng.standard_normal(shape) * 0.5).astype(np.float32) for _ in range(dim)] for _ in range(SNAPSHOTS)]
    stored = [[W.round_storage(p, ("f32", "bf16", "f16")[storage]) for p in s] for s in snaps]
    base = dict(Space=0 if dim == 3 else 1, Integrator=1, WindfieldMode=1, DeltaT=0.25, DataTimeDistance=1.0,
                GridScale=[1.0] * dim, Offset=[0.0] * dim, SaveInterval=0, MaximumSimulationTime=SNAPSHOTS - 1.0)
    srv = capi.Server(capi.settings_from_reference(base, storage=storage), SNAPSHOTS, shape, hbm_budget=4 << 20)
    for k, s in enumerate(snaps):
        srv.set_snapshot(k, s)
    srv.start()
    reqs = [dict(seeds=rng.uniform(0, shape[::-1], (int(n), dim)).astype(np.float32), k0=int(k0), steps=int(m), rk4=r)
            for n, k0, m, r in [(1, 0, 27, 1), (33, 5, 9, 0), (700, 2, 26, 1), (257, 13, 1, 1), (1025, 26, 2, 0)]]
    for again in range(2):   # the second round finds pairs built
        ids = [srv.submit(r["seeds"], 0.25 * r["k0"], r["steps"], r["rk4"]) for r in reqs]
        for rid, r in zip(ids, reqs):
            assert srv.wait(rid, 60.0) == capi.GR_REQ_DONE
            pos, st, info = srv.result(rid)
            srv.release(rid)
            ref = orc.run(orc.settings(**dict(base, Integrator=r["rk4"])), orc.Inputs(wind=stored, seeds=r["seeds"]),
                          precision="f32", start_step=r["k0"], step_limit=r["k0"] + r["steps"])
            assert np.array_equal(st, ref["status"])
            assert np.array_equal(pos, ref["trajectories"][:, -1])
    assert (srv.stats().h2d_bytes > sum(2 * r["seeds"].nbytes for r in reqs) * 3) == (resident == "0")
    srv.close()
