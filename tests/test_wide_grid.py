"""Grids with an axis of 2^22 nodes and more (GPU), where float32 coordinates leave the range of the fast cell
arithmetic: the engine in either layout, gr_advance_noalloc and the request server, with particles on both sides of
2^22, bit for bit against the float32 oracle."""
import numpy as np
import pytest

from oracle import oracle as orc
from pygranite_b200 import capi
from pygranite_b200 import workloads as W
from tests import harness as H

pytestmark = pytest.mark.gpu

NX, WINDOWS, PER_WINDOW = 4_200_000, 2, 4
SHAPES = {2: (2, NX), 3: (1, 2, NX)}


@pytest.fixture(scope="module", params=[(2, 0), (2, 1), (3, 0)], ids=["2d-f32", "2d-bf16", "3d-f32"])
def problem(request):
    dim, storage = request.param
    rng = np.random.default_rng(dim + storage)
    shape = SHAPES[dim]
    size = (4.0, 0.02, 0.02)      # cells a step: positions beyond 2^22 are multiples of 0.5
    wind = [[rng.standard_normal(shape, dtype=np.float32) * np.float32(size[k]) for k in range(dim)]
            for _ in range(WINDOWS + 1)]
    stored = [[W.round_storage(p, ("f32", "bf16")[storage]) for p in s] for s in wind]
    x = np.concatenate([2.0 ** 22 + rng.uniform(-60, 60, 100), rng.uniform(2.0 ** 22, NX, 100), NX - rng.uniform(0, 20, 30),
                        rng.uniform(0, 40, 30), rng.uniform(0, NX, 40)])
    seeds = np.stack([x] + [rng.uniform(0.1, s - 0.1, x.size) for s in shape[-2::-1]], axis=1).astype(np.float32)
    settings = dict(Space=0 if dim == 3 else 1, WindfieldMode=1, DeltaT=1.0, DataTimeDistance=float(PER_WINDOW),
                    GridScale=[1.0] * dim, Offset=[0.0] * dim, SaveInterval=0,
                    MaximumSimulationTime=float(PER_WINDOW * WINDOWS))
    ref = {rk4: orc.run(orc.settings(**dict(settings, Integrator=rk4)), orc.Inputs(wind=stored, seeds=seeds),
                        precision="f32") for rk4 in (0, 1)}
    assert (ref[1]["status"] == 0).sum() > 150
    return settings, storage, shape, wind, seeds, ref


@pytest.mark.parametrize("rk4", [0, 1])
@pytest.mark.parametrize("layout", [0, 1])
def test_engine(problem, layout, rk4):
    settings, storage, shape, wind, seeds, ref = problem
    e = capi.Engine(capi.settings_from_reference(dict(settings, Integrator=rk4), ring_slots=WINDOWS + 1,
                                                 storage=storage, layout=layout))
    e.set_seeds(seeds)
    for k, s in enumerate(wind):
        e.load_windfield(k, s)
    e.run(lambda k: 1 if k <= WINDOWS else 0)
    H.assert_same(e.results(), ref[rk4])
    e.close()


@pytest.mark.parametrize("rk4", [0, 1])
def test_server(problem, rk4):
    settings, storage, shape, wind, seeds, ref = problem
    srv = capi.Server(capi.settings_from_reference(settings, storage=storage), WINDOWS + 1, shape, hbm_budget=4 << 20)
    for k, s in enumerate(wind):
        srv.set_snapshot(k, s)
    srv.start()
    for again in range(2):
        rid = srv.submit(seeds, 0.0, PER_WINDOW * WINDOWS, rk4)
        assert srv.wait(rid, 60.0) == capi.GR_REQ_DONE
        pos, st, _ = srv.result(rid)
        srv.release(rid)
        assert np.array_equal(st, ref[rk4]["status"])
        assert np.array_equal(pos, ref[rk4]["trajectories"][:, -1])
    srv.close()


def test_server_from_host_memory(problem, monkeypatch):
    monkeypatch.setenv("GR_SERVE_RESIDENT", "0")
    test_server(problem, 1)


def test_noalloc(problem):
    import torch
    settings, storage, shape, wind, seeds, _ = problem
    if storage != 0:
        pytest.skip("float32 storage only")
    dim = len(shape)
    node = [np.stack(s + ([np.zeros_like(s[0])] if dim == 3 else []), axis=-1) for s in wind[:2]]
    dev = [torch.from_numpy(a).cuda() for a in node]
    state = torch.zeros((4, len(seeds)), device="cuda")
    state[:dim] = torch.from_numpy(seeds.T.copy()).cuda()
    torch.cuda.synchronize()
    row = [state[k].data_ptr() for k in range(4)]
    capi.advance_noalloc(capi.settings_from_reference(dict(settings, Integrator=1)), shape, dev[0].data_ptr(),
                         dev[1].data_ptr(), 0.0, float(PER_WINDOW), 0.0, PER_WINDOW, row[0], row[1],
                         row[2] if dim == 3 else None, row[3], len(seeds))
    torch.cuda.synchronize()
    ref = orc.run(orc.settings(**dict(settings, Integrator=1)), orc.Inputs(wind=wind, seeds=seeds), precision="f32",
                  step_limit=PER_WINDOW)
    assert np.array_equal(state[3].view(torch.int32).cpu().numpy(), ref["status"])
    assert np.array_equal(state[:dim].T.cpu().numpy(), ref["trajectories"][:, -1])
