"""Inputs that a call copies to the device are there before its kernels read them (GPU).  The kernels run on streams that
do not wait for the default stream, and a copy from pageable memory or on the device may still be under way when the
copying call returns."""
import numpy as np
import pytest

from oracle import oracle as orc
from pygranite_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", [0, 1])
def test_server_field_from_pageable_planes(storage):
    shape, snapshots = (40, 60, 70), 12            # planes of 672 KB
    rng = np.random.default_rng(8)
    wind = [[(rng.standard_normal(shape) * 0.5).astype(np.float32) for _ in range(3)] for _ in range(snapshots)]
    base = dict(Space=0, Integrator=1, WindfieldMode=1, DeltaT=0.25, DataTimeDistance=1.0, GridScale=[1.0] * 3,
                Offset=[0.0] * 3, SaveInterval=0, MaximumSimulationTime=snapshots - 1.0)
    seeds = rng.uniform(0, shape[::-1], (3000, 3)).astype(np.float32)
    from pygranite_b200 import workloads as W
    stored = [[W.round_storage(p, ("f32", "bf16")[storage]) for p in s] for s in wind]
    ref = orc.run(orc.settings(**base), orc.Inputs(wind=stored, seeds=seeds), precision="f32")
    wrong = 0
    for again in range(10):
        srv = capi.Server(capi.settings_from_reference(base, storage=storage), snapshots, shape, hbm_budget=4 << 20)
        for k, s in enumerate(wind):
            srv.set_snapshot(k, s)
        srv.start()
        rid = srv.submit(seeds, 0.0, 4 * (snapshots - 1), 1)
        assert srv.wait(rid, 60.0) == capi.GR_REQ_DONE
        pos, st, _ = srv.result(rid)
        srv.close()
        wrong += not (np.array_equal(st, ref["status"]) and np.array_equal(pos, ref["trajectories"][:, -1]))
    assert wrong == 0


def still_engine(n, **kw):
    """An engine whose particles keep their seeds: no wind, so every step ends at once."""
    e = capi.Engine(capi.settings_from_reference(
        dict(Space=0, Integrator=0, WindfieldMode=1, DeltaT=1.0, DataTimeDistance=1.0, GridScale=[1.0] * 3, Offset=[0.0] * 3,
             SaveInterval=0, MaximumSimulationTime=1.0), ring_slots=3, **kw))
    for k in range(2):
        e.load_windfield(k, [np.zeros((4, 4, 4), np.float32)] * 3)
    return e


@pytest.mark.parametrize("n", [10_000, 1_000_000, 12_000_000])
def test_device_seeds(n):
    import torch
    e = still_engine(n)
    a = torch.rand((n, 3), device="cuda") * 2 + 1
    b = torch.rand((n, 3), device="cuda") * 2 + 1
    torch.cuda.synchronize()
    ref = [a.cpu().numpy(), b.cpu().numpy()]
    for k, s in enumerate([a, b] * 3):
        e.set_seeds_device(s.data_ptr(), n, 3)
        e.run(lambda k: 0)
        assert np.array_equal(e.final_positions(), ref[k & 1]), k
    e.close()


@pytest.mark.parametrize("n", [4_000, 100_000, 3_000_000])
def test_host_seeds_of_a_batch(n):
    rng = np.random.default_rng(n)
    e = still_engine(n)
    seeds = [rng.uniform(1, 3, (n, 3)).astype(np.float32) for _ in range(2)]
    e.set_seeds(seeds[0])
    batch = capi.Batch([e])
    for k in range(8):
        e.set_seeds(seeds[k & 1])
        batch.run()
        assert np.array_equal(e.final_positions(), seeds[k & 1]), k
    batch.close()
    e.close()
