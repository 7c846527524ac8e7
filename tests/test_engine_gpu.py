"""The Evaluator's recorded calls (CUDA graphs whose kernel launches are chained to one another) against its eager
calls and the CPU checker: the same numbers after many back-to-back replays, and a replay sees the positions that
are in the buffers at that time. What a calculator does per call: ai2pot/models/potential_utils.py:217-268."""
import numpy as np
import pytest
import torch

import util
from ai2pot_b200 import engine, synth

pytestmark = pytest.mark.gpu


def _workload(kind, n):
    if kind == "mtp":
        return synth.g1(util.tables(16), n=n), torch.float64, 1e-10
    return synth.g2(n=n), torch.float32, 1e-5


def _moved(w, seed):
    rng = np.random.default_rng(seed)
    return (w["coords"] + rng.normal(0, 0.05, w["coords"].shape)).astype(w["coords"].dtype)


def _host(out):
    return tuple(t.detach().cpu().numpy().copy() for t in out)


def _close(a, b, tol):
    for x, y in zip(a, b):
        assert util.relerr(x, y) < tol


@pytest.mark.parametrize("kind", ["mtp", "nep"])
def test_replay_equals_eager_and_checker(kind, checkers):
    w, dt, tol = _workload(kind, 10)          # 1,000 atoms
    ev = engine.Evaluator(w["model"], w["cell"], w["types"], w["rcut"], w["umax"], dt)
    pos = [np.ascontiguousarray(w["coords"]), _moved(w, 5), _moved(w, 6)]
    coords = torch.from_numpy(pos[0]).to(dt).cuda()
    eager = []
    for p in pos:
        coords.copy_(torch.from_numpy(p).to(dt))
        eager.append(_host(ev.compute(coords)))
    assert int(ev.status.cpu()[1]) == 0
    # the CPU code on the first configuration
    chk = checkers.get("ref") or checkers["oracle"]
    nn, fn, rc, ty, mx = chk.nblist(w["cell"], w["types"], pos[0], w["rcut"], w["umax"])
    nb = synth.batch_from_nblist(nn, fn, rc, ty, 3)
    ref = chk.mtp_efv(w["model"], nb) if kind == "mtp" else chk.nep_efv(w["model"], nb)
    _close(eager[0], ref[:3], tol)

    assert ev.capture(coords)
    for k in (1, 2, 0):
        coords.copy_(torch.from_numpy(pos[k]).to(dt))
        for _ in range(20):                    # back to back, nothing in between: the outputs are rebuilt by every replay
            out = ev.replay()
        _close(_host(out), eager[k], tol)

    # the whole call as one graph: pinned host positions in, one pinned host buffer out
    h_in = torch.empty_like(coords, device="cpu").pin_memory()
    h_out = torch.empty(ev.outbuf.shape, dtype=dt).pin_memory()
    h_in.copy_(torch.from_numpy(pos[0]).to(dt))
    assert ev.capture_io(coords, h_in, h_out)
    n = len(w["types"])
    for k in (2, 0, 1):
        h_in.copy_(torch.from_numpy(pos[k]).to(dt))
        h_out.fill_(float("nan"))
        for _ in range(5):
            ev.replay_io()
        torch.cuda.synchronize()
        got = (h_out[0:1].numpy(), h_out[16:16 + 3 * n].numpy().reshape(1, n, 3), h_out[1:10].numpy().reshape(1, 9))
        _close(got, eager[k], tol)


@pytest.mark.parametrize("kind", ["mtp", "nep"])
def test_ordinary_launches_give_the_same(kind, monkeypatch):
    """AI2B_CHAIN=0 switches the chained launches off: same numbers either way."""
    w, dt, tol = _workload(kind, 8)
    ev = engine.Evaluator(w["model"], w["cell"], w["types"], w["rcut"], w["umax"], dt)
    coords = torch.from_numpy(np.ascontiguousarray(w["coords"])).to(dt).cuda()
    chained = _host(ev.compute(coords))
    monkeypatch.setenv("AI2B_CHAIN", "0")
    plain = _host(ev.compute(coords))
    monkeypatch.delenv("AI2B_CHAIN")
    again = _host(ev.compute(coords))
    _close(plain, chained, tol)
    _close(again, chained, tol)


@pytest.mark.parametrize("n", [8, 14])
def test_build_and_evaluation_share_scratch(n):
    """One buffer as the scratch of the neighbour build and of the evaluation, below and above the size from which atoms are binned
    by several launches: the evaluation's set-up does not run ahead of the build then."""
    w, dt, tol = _workload("nep", n)
    ev = engine.Evaluator(w["model"], w["cell"], w["types"], w["rcut"], w["umax"], dt)
    coords = torch.from_numpy(np.ascontiguousarray(w["coords"])).to(dt).cuda()
    apart = _host(ev.compute(coords))
    ev.ws = ev.nb_ws = torch.empty(max(ev.ws.numel(), ev.nb_ws.numel()), dtype=torch.uint8, device="cuda")
    ev._filled = None
    _close(_host(ev.compute(coords)), apart, tol)


@pytest.mark.parametrize("n", [8, 14])
@pytest.mark.parametrize("where", ["nb_ws", "coords"])
def test_results_in_memory_that_the_build_reads(n, where):
    """Energy, forces and virial in the build's scratch or over the positions: both are free once the rows stand, so the call
    is answered, and its set-up, which zeroes them, waits for the build."""
    w, dt, tol = _workload("nep", n)
    ev = engine.Evaluator(w["model"], w["cell"], w["types"], w["rcut"], w["umax"], dt)
    coords = torch.from_numpy(np.ascontiguousarray(w["coords"])).to(dt).cuda()
    apart = _host(ev.compute(coords))
    memory = ev.nb_ws.view(-1) if where == "nb_ws" else coords.view(-1).view(torch.uint8)
    kept = ev.out
    for k in range(3):      # one at a time, at the beginning of the memory
        moved = memory[:kept[k].numel() * kept[k].element_size()].view(dt).view(kept[k].shape)
        ev.out = kept[:k] + (moved,) + kept[k + 1:]
        _close(_host(ev.compute(coords)), apart, tol)
        coords.copy_(torch.from_numpy(np.ascontiguousarray(w["coords"])).to(dt))


@pytest.mark.parametrize("n", [8, 14])
def test_status_words_in_the_scratch_of_the_evaluation(n):
    """The build's status words where the evaluation lays its model table: they are the build's until the rows stand, and the memory is
    the evaluation's after that. (Negative values: the build would raise them to its counts.)"""
    w, dt, tol = _workload("nep", n)
    w["model"]["coeffs"] = -np.abs(w["model"]["coeffs"])
    ev = engine.Evaluator(w["model"], w["cell"], w["types"], w["rcut"], w["umax"], dt)
    coords = torch.from_numpy(np.ascontiguousarray(w["coords"])).to(dt).cuda()
    apart = _host(ev.compute(coords))
    ev.lists = ev.lists[:3] + (ev.ws[256:264].view(torch.int32),)      # (the table follows the offsets of one structure)
    ev._filled = None
    _close(_host(ev.compute(coords)), apart, tol)


@pytest.mark.parametrize("kind", ["mtp", "nep"])
def test_changed_attributes_take_effect(kind):
    """Cell, cutoff, row width and model may be edited or assigned between calls (a variable-cell relaxation does): the next
    call is that of an Evaluator made with them. A recorded call goes on as it was recorded."""
    w, dt, tol = _workload(kind, 8)
    make = lambda model, cell, rcut: engine.Evaluator(model, cell, w["types"], rcut, 96, dt)
    cell, model = np.array(w["cell"]), w["model"]
    ev = engine.Evaluator(model, cell, w["types"], w["rcut"], w["umax"], dt)
    coords = torch.from_numpy(np.ascontiguousarray(w["coords"])).to(dt).cuda()
    before = _host(ev.compute(coords))
    assert ev.capture(coords)

    def same(want):
        _close(_host(ev.compute(coords)), want, tol)
        _close(_host(ev.evaluate(ev.build_list(coords))), want, tol)      # the two steps of a call one by one

    strained = cell * cell.dtype.type(1.03)
    want = _host(make(model, strained, w["rcut"]).compute(coords))
    assert util.relerr(want[0], before[0]) > 10 * tol
    ev.cell[:] = strained                     # edited in place
    same(want)
    sheared = strained.copy()
    sheared[1, 0] += 0.5
    ev.cell = sheared                         # another array
    same(_host(make(model, sheared, w["rcut"]).compute(coords)))
    ev.rcut, ev.umax = 0.75 * w["rcut"], 96   # rows of another width
    same(_host(make(model, sheared, 0.75 * w["rcut"]).compute(coords)))
    assert ev.lists[1].shape[1] == 96 and int(ev.status.cpu()[0]) <= 96
    other = dict(model, coeffs=model["coeffs"] * model["coeffs"].dtype.type(0.9))
    ev.model["coeffs"] = 0.9 * ev.model["coeffs"]
    same(_host(make(other, sheared, 0.75 * w["rcut"]).compute(coords)))
    _close(_host(ev.replay()), before, tol)
    # a tensor that the kernels cannot read is refused, also where its address is that of the last call's
    for name, bad in (("coeffs", ev.model["coeffs"].cpu()), ("q_scaler", ev.model["q_scaler"].expand(2, -1).t()[:, 0][::2])):
        good, ev.model[name] = ev.model[name], bad
        with pytest.raises(engine.capi.Ai2bError):
            ev.compute(coords)
        ev.model[name] = good
    for wrong in (np.eye(3)[:2], np.ones(3)):
        good, ev.cell = ev.cell, wrong
        with pytest.raises(ValueError):
            ev.compute(coords)
        ev.cell = good
    ev.cell = list(map(list, sheared))
    same(_host(make(other, sheared, 0.75 * w["rcut"]).compute(coords)))


def test_positions_that_do_not_fit_are_refused():
    """The buffers of an Evaluator are those of its structure and type."""
    w, dt, _ = _workload("nep", 6)
    ev = engine.Evaluator(w["model"], w["cell"], w["types"], w["rcut"], w["umax"], dt)
    coords = torch.from_numpy(np.ascontiguousarray(w["coords"])).to(dt).cuda()
    for bad in (coords.double(), coords[:-1], torch.cat([coords, coords[:1]]), coords.cpu()):
        for call in (ev.compute, ev.build_list):
            with pytest.raises(engine.capi.Ai2bError):
                call(bad)
    strided = torch.empty(ev.n, 4, dtype=dt, device="cuda")[:, :3].copy_(coords)
    _close(_host(ev.compute(strided)), _host(ev.compute(coords)), 1e-5)


@pytest.mark.parametrize("kind,natoms,ntypes", [("mtp", 216, 3), ("nep", 216, 3), ("nep", 2197, 3), ("mtp", 2197, 3), ("nep", 2197, 17), ("nep", 300000, 3)])
def test_launch_counts(kind, natoms, ntypes):
    """launches_per_step() against the nodes of a recorded call: few atoms, several binning launches, the general NEP kernel,
    and (sparse cell, more than 8,192 bins) a scan of its own."""
    import ctypes as C
    rng = np.random.default_rng(natoms)
    spacing = 3.0 if natoms < 10000 else 6.0
    edge = int(np.ceil(natoms ** (1.0 / 3.0) - 1e-9))
    dt = torch.float64 if kind == "mtp" else torch.float32
    npdt = np.float64 if kind == "mtp" else np.float32
    cell, pos = synth.cubic_lattice(edge, spacing, 0.1, rng, npdt, nocc=natoms)
    model = synth.mtp_model(util.tables(10), ntypes, rng, npdt, 5.0, 0.5) if kind == "mtp" else synth.nep_model(ntypes, rng, npdt)
    ev = engine.Evaluator(model, cell, rng.integers(0, ntypes, natoms).astype(np.int32), 5.0 if kind == "mtp" else 6.0, 64, dt)
    coords = torch.from_numpy(pos).cuda()
    ev.compute(coords)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        ev.compute(coords)
    nodes = C.c_size_t(0)
    assert C.CDLL("libcudart.so.12").cudaGraphGetNodes(C.c_void_p(graph.raw_cuda_graph()), None, C.byref(nodes)) == 0
    assert ev.launches_per_step() == nodes.value
