"""What users of this package have it do, as cases that can be timed and compared.

Paths (the public entry points that a pass goes through):
  evaluate  a calculator: positions in, energy / forces / virial out (engine.Evaluator: compute() call by call, or the
            whole call with pinned host buffers recorded once and replayed)
  train     one step of potential fitting: the loss op of fromcc on a resident padded batch, then backward() to the
            model parameters
  md        a molecular-dynamics host: double positions of local and ghost atoms in host memory in, forces out
            (capi.MdSession.compute)
  list      the reference's host neighbour list, numpy in and numpy out (fromcc.nblist.find_info4mlff)
  frames    neighbour tensors of many small frames before training (capi.nblist_build_batch + row sort)

Sizes, models and cutoffs are those of ai2pot_b200/synth.py, of bench.py and of the tests. Every structure, model and
target comes from the seed."""
import math

import numpy as np
import torch

from ai2pot_b200 import capi, synth, tables
from ai2pot_b200.engine import Evaluator

SPACING = 3.0        # lattice constant of synth's simple cubic structures
RCUT = {"mtp06": 5.0, "mtp10": 5.0, "mtp16": 6.0, "nep": 6.0}


def listed():
    return [
        # the smallest structure: a relaxation or a phonon displacement, where latency counts
        {"name": "evaluate_mtp10_f64_216", "path": "evaluate", "model": "mtp10", "dtype": "f64", "natoms": 216, "call": "compute"},
        # a small cell that is not a full lattice, driven from the host step after step by a recorded call
        {"name": "evaluate_nep_f32_1157_io", "path": "evaluate", "model": "nep", "dtype": "f32", "natoms": 1157, "call": "replay_io"},
        # linear MTP in double precision
        {"name": "evaluate_mtp16_f64_13824", "path": "evaluate", "model": "mtp16", "dtype": "f64", "natoms": 13824, "call": "compute"},
        # NEP in single precision on the same structure
        {"name": "evaluate_nep_f32_13824", "path": "evaluate", "model": "nep", "dtype": "f32", "natoms": 13824, "call": "compute"},
        # the largest system, a decorated cubic crystal with four atoms per cell
        {"name": "evaluate_nep_f32_1048576", "path": "evaluate", "model": "nep_crystal", "dtype": "f32", "natoms": 1048576, "call": "compute"},
        # a training step, forward and backward, on a ragged batch
        {"name": "train_mtp16_f64_64", "path": "train", "model": "mtp16", "dtype": "f64", "batch": 64, "nmin": 64, "nmax": 256},
        {"name": "train_nep_f32_64", "path": "train", "model": "nep", "dtype": "f32", "batch": 64, "nmin": 64, "nmax": 256},
        # a mini-batch of small cells in single precision
        {"name": "train_mtp10_f32_8", "path": "train", "model": "mtp10", "dtype": "f32", "batch": 8, "nmin": 20, "nmax": 40},
        # one force call of an MD code: the ghost atoms out to the cutoff come with the local ones
        {"name": "md_nep_13824", "path": "md", "model": "nep", "natoms": 13824},
        {"name": "md_mtp16_3001", "path": "md", "model": "mtp16", "natoms": 3001},
        # the neighbour list that the reference's calculators and dataset ask for, rows sorted by distance
        {"name": "list_f64_2197", "path": "list", "dtype": "f64", "natoms": 2197},
        # the pre-training pass over a dataset
        {"name": "frames_f64_64", "path": "frames", "dtype": "f64", "batch": 64, "nmin": 64, "nmax": 256},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    path = rng.choice(["evaluate", "evaluate", "evaluate", "train", "train", "md", "md", "list", "frames"])
    if path == "evaluate":
        model = rng.choice(["mtp06", "mtp10", "mtp16", "nep", "nep", "nep_crystal"])
        dtype = rng.choice(["f64", "f32"]) if model.startswith("mtp") else rng.choice(["f32", "f32", "f64"])
        top = {"mtp06": 131072, "mtp10": 131072, "mtp16": 100000, "nep": 300000, "nep_crystal": 700000}[model]
        if model.startswith("nep") and dtype == "f64":
            top = 100000
        return {"path": path, "model": model, "dtype": dtype, "natoms": size(200 if model != "nep_crystal" else 2000, top),
                "call": rng.choice(["compute", "compute", "replay_io"])}
    if path == "train":
        nmin = size(16, 100)
        return {"path": path, "model": rng.choice(["mtp10", "mtp16", "nep", "nep"]), "dtype": rng.choice(["f64", "f32"]),
                "batch": size(4, 64), "nmin": nmin, "nmax": size(nmin + 1, 256)}
    if path == "md":
        return {"path": path, "model": rng.choice(["nep", "nep", "mtp10", "mtp16"]), "natoms": size(500, 13824)}
    if path == "list":
        return {"path": path, "dtype": "f64", "natoms": size(216, 2197)}
    nmin = size(16, 100)
    return {"path": path, "dtype": "f64", "batch": size(4, 64), "nmin": nmin, "nmax": size(nmin + 1, 256)}


def _np_dtype(case):
    return np.float64 if case.get("dtype") == "f64" else np.float32


def _torch_dtype(case):
    return torch.float64 if case.get("dtype") == "f64" else torch.float32


def _rcut(case):
    return RCUT.get(case.get("model", "nep"), 6.0)


def _model(name, rng, dtype):
    if name.startswith("nep"):
        m = synth.nep_model(3, rng, dtype)
    else:
        m = synth.mtp_model(tables.load(int(name[3:])), 3, rng, dtype, RCUT[name], 0.5)
    m["type_bias"] = rng.normal(0, 0.1, 3).astype(dtype)
    m["q_scaler"] = rng.uniform(0.5, 1.5, len(m["q_scaler"])).astype(dtype)
    return m


def _structure(case, rng, dtype):
    """cell, positions, types, umax. A count that fills no lattice leaves the last layers of the cell open."""
    n = case["natoms"]
    if case.get("model") == "nep_crystal":
        edge = math.ceil((n / 4) ** (1.0 / 3.0) - 1e-9)
        g = np.arange(edge, dtype=np.float64) * 6.0
        org = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 1, 3)
        basis = np.array([[0, 0, 0], [.5, .5, .5], [.5, 0, 0], [0, .5, .5]]) * 6.0
        pos = (org + basis[None]).reshape(-1, 3)[:n]
        types = np.tile(np.array([0, 0, 2, 2], np.int32), edge ** 3)[:n]
        types[(types == 0) & (rng.random(n) < 0.2)] = 1
        pos = pos + rng.normal(0, 0.1, pos.shape)
        return (np.eye(3) * (edge * 6.0)).astype(dtype), pos.astype(dtype), types, 32
    edge = math.ceil(n ** (1.0 / 3.0) - 1e-9)
    cell, pos = synth.cubic_lattice(edge, SPACING, 0.1, rng, dtype, nocc=n)
    types = rng.choice(3, size=n, p=np.array([2, 2, 5]) / 9.0).astype(np.int32)
    return cell, pos, types, 64


def _frames(case, rng):
    """Padded host arrays of a ragged set of small cells, the ends of its size range among them."""
    B, lo, hi = case["batch"], case["nmin"], case["nmax"]
    sizes = rng.integers(lo, hi + 1, B)
    sizes[0], sizes[-1] = lo, hi
    cells, coords = np.zeros((B, 3, 3)), np.zeros((B, hi, 3))
    types = np.zeros((B, hi), np.int32)
    for b, n in enumerate(sizes):
        n = int(n)
        edge = math.ceil(n ** (1.0 / 3.0) - 1e-9)
        cells[b], coords[b, :n] = synth.cubic_lattice(edge, float(rng.uniform(2.8, 3.2)), 0.15, rng, nocc=n)
        types[b, :n] = rng.integers(0, 3, n)
    return cells, sizes.astype(np.int32), coords, types


def _prepare_evaluate(case, rng):
    dt, npdt = _torch_dtype(case), _np_dtype(case)
    cell, pos, types, umax = _structure(case, rng, npdt)
    model = _model(case["model"], rng, npdt)
    ev = Evaluator(model, cell, types, _rcut(case), umax, dt)
    coords = torch.from_numpy(np.ascontiguousarray(pos)).cuda()
    state = {"case": case, "ev": ev, "coords": coords}
    if case["call"] == "replay_io":
        state["h_in"] = torch.from_numpy(np.ascontiguousarray(pos)).pin_memory()
        state["h_out"] = torch.zeros(ev.outbuf.shape, dtype=dt).pin_memory()
        ev.outbuf.zero_()                 # the gap between the virial and the forces is not written by a call
        ev.compute(coords)
        if not ev.capture_io(coords, state["h_in"], state["h_out"]):
            raise RuntimeError("the call could not be recorded")
    return state


def _prepare_train(case, rng):
    from ai2pot_b200 import fromcc
    dt, npdt = _torch_dtype(case), _np_dtype(case)
    cells, binum, coords, types = _frames(case, rng)
    model = _model(case["model"], rng, npdt)
    dev = lambda a, t=None: torch.from_numpy(np.ascontiguousarray(a)).to("cuda", t)
    B, npad = types.shape
    nb = capi.nblist_build_batch(cells.astype(npdt), dev(binum), dev(coords, dt), _rcut(case), 64)
    if int(nb["status"][1]):
        raise RuntimeError("more than 64 neighbours")
    zbl = torch.zeros(36, dtype=dt, device="cuda")
    targets = (dev(rng.normal(0, 1, B), dt), dev(rng.normal(0, 1, (B, npad, 3)), dt), dev(rng.normal(0, 1, (B, 9)), dt))
    lists = (nb["binum"], nb["bilist"], nb["bnumneigh"], nb["bfirstneigh"], nb["brcs"], dev(types), dev(np.arange(3, dtype=np.int32)), 0)
    if case["model"] == "nep":
        params = [dev(model[k], dt).requires_grad_(True) for k in ("coeffs", "w0", "b0", "w1", "type_bias")]
        op = fromcc.nepToLossOp
        args = (1.0, 1.0, 1.0, *targets, model["chebyshev_size"], model["n_radial"], model["n_angular"], model["l_max"], *params, *lists,
                model["rmax_radial"], model["rmax_angular"], dev(model["q_scaler"], dt), 0.0, 0.0, zbl, zbl)
    else:
        params = [dev(model[k], dt).requires_grad_(True) for k in ("coeffs", "linear_coeffs", "type_bias")]
        op, tb = fromcc.linearMtpToLossOp, model["tables"]
        args = (1.0, 1.0, 1.0, *targets, model["chebyshev_size"], model["scaling"], *params, tb["alpha_moments_count"],
                dev(tb["alpha_index_basic"]), dev(tb["alpha_index_times"]), dev(tb["alpha_moment_mapping"]), tb["nmus"], *lists,
                model["rmax"], model["rmin"], dev(model["q_scaler"], dt), 0.0, 0.0, zbl, zbl)
    return {"case": case, "op": op, "args": args, "params": params}


def _ghosts(case):
    """Ghost atoms of an MD host: the periodic images within the cutoff and a skin of 2.0 of the box."""
    n = case["natoms"]
    edge = math.ceil(n ** (1.0 / 3.0) - 1e-9) * SPACING
    return min(26 * n, int(n * ((1 + 2 * (_rcut(case) + 2.0) / edge) ** 3 - 1)))


def _prepare_md(case, rng):
    cell, pos, types, umax = _structure(case, rng, np.float64)
    rcut = _rcut(case)
    L = np.diag(cell)
    x = np.mod(pos, L)
    shifts = np.array([(i, j, k) for i in (-1, 0, 1) for j in (-1, 0, 1) for k in (-1, 0, 1) if (i, j, k) != (0, 0, 0)]) * L
    images = (x[None] + shifts[:, None]).reshape(-1, 3)
    outside = np.maximum(-images, images - L).max(axis=1)          # how far outside the box
    nghost = _ghosts(case)                                          # the same count for every seed
    order = np.argsort(outside, kind="stable")[:nghost + 1]
    if len(order) > nghost and outside[order[-1]] < rcut:
        raise RuntimeError("ghost atoms within the cutoff are missing")
    ghosts = order[:nghost]
    xa = np.ascontiguousarray(np.concatenate([x, images[ghosts]]))
    ta = np.ascontiguousarray(np.concatenate([types, np.tile(types, 26)[ghosts]]).astype(np.int32))
    model = _model(case["model"], rng, np.float32)
    prog = capi.MtpProgram(model["tables"]) if model["kind"] == "mtp" else None
    return {"case": case, "session": capi.MdSession(model, umax, prog), "nlocal": len(x), "nghost": nghost, "x": xa, "types": ta}


def _prepare_list(case, rng):
    cell, pos, types, umax = _structure(case, rng, _np_dtype(case))
    return {"case": case, "args": (cell, types, pos, 6.0, umax, True, [True, True, True], True)}


def _prepare_frames(case, rng):
    cells, binum, coords, _ = _frames(case, rng)
    return {"case": case, "cells": cells, "binum": torch.from_numpy(binum).cuda(), "coords": torch.from_numpy(coords).cuda()}


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    return {"evaluate": _prepare_evaluate, "train": _prepare_train, "md": _prepare_md, "list": _prepare_list,
            "frames": _prepare_frames}[case["path"]](case, rng)


def run(state):
    path = state["case"]["path"]
    if path == "evaluate":
        if "h_in" in state:
            state["ev"].replay_io()
            return state["h_out"]
        return state["ev"].compute(state["coords"])
    if path == "train":
        for p in state["params"]:
            p.grad = None
        out = state["op"](*state["args"])
        out[0].mean().backward()
        return [o.detach() for o in out] + [p.grad for p in state["params"]]
    if path == "md":
        return state["session"].compute(state["nlocal"], state["nghost"], state["x"], state["types"])
    if path == "list":
        from ai2pot_b200.fromcc import nblist
        return nblist.find_info4mlff(*state["args"])
    nb = capi.nblist_build_batch(state["cells"], state["binum"], state["coords"], 6.0, 64)
    n = nb["bnumneigh"].numel()
    capi.sort_rows_by_distance(nb["bnumneigh"].view(n), nb["bfirstneigh"].view(n, 64), nb["brcs"].view(n, 64, 3))
    return nb


def _neighbours(case):
    """Mean neighbour counts of the structures above: within the cutoff, within the angular cutoff of NEP (4.0)."""
    if case.get("model") == "nep_crystal":
        return 16.9, 2.2
    return (29.0, 6.5) if _rcut(case) == 6.0 else (18.7, 6.5)


def _flops_per_atom(case, training=False):
    """Floating-point work of energy, forces and virial per atom (a fused multiply-add counts as two)."""
    nn, nn_a = _neighbours(case)
    cs = 8
    if case["model"].startswith("nep"):
        n, neurons, nd = 4, 30, 20
        fl = (nn * (9 * cs + 20 + 4 * n * cs + 4 * n + 12) + nn_a * (9 * cs + 20 + 4 * n * cs + 384 + 528 * n) + 144 * n
              + 4 * neurons * nd + 20 * neurons)
        return 3 * fl if training else fl
    tb = tables.load(int(case["model"][3:]))
    nbasic, nt, ns = (len(tb[k]) for k in ("alpha_index_basic", "alpha_index_times", "alpha_moment_mapping"))
    kmax = int(tb["alpha_index_basic"][:, 1:].sum(1).max())
    radial = 9 * cs + 20 + 4 * tb["nmus"] * cs
    fl = nn * (radial + 4 * kmax + 4 + 29 * nbasic) + 9 * nt + 4 * ns
    return fl + nn * (55 * nbasic + radial) + 18 * nt + 6 * ns if training else fl


def work(case):
    s = 8 if case.get("dtype") == "f64" else 4
    path = case["path"]
    if path == "evaluate":
        n = case["natoms"]
        return {"bytes": n * (6 * s + 4), "flops": n * _flops_per_atom(case)}
    if path == "md":       # double positions and types of local and ghost atoms in, double forces out
        n = case["natoms"]
        return {"bytes": (n + _ghosts(case)) * 52, "flops": n * _flops_per_atom(case)}
    if path == "list":     # positions in; padded rows, counts, centre list and types out
        n = case["natoms"]
        return {"bytes": n * (3 * s + 64 * (4 + 3 * s) + 16), "flops": n * 27 * 8 * 10}
    natoms = case["batch"] * (case["nmin"] + case["nmax"]) / 2
    slots = case["batch"] * case["nmax"]
    if path == "frames":
        return {"bytes": slots * (3 * s + 64 * (4 + 3 * s) + 8), "flops": natoms * 27 * 8 * 10}
    nn = _neighbours(case)[0]      # the filled part of the rows, targets and types in; loss and gradients out
    return {"bytes": natoms * (nn * (4 + 3 * s) + 3 * s + 12), "flops": natoms * _flops_per_atom(case, True)}


def tolerance(case):
    if case["path"] in ("list", "frames"):
        return "exact"     # rows sorted by distance (no ties in double precision), and the distances are defined bit for bit
    return {"rel": 1e-11} if case.get("dtype") == "f64" else {"rel": 1e-5}
