"""Parity of the CUDA linear-MTP path (through the C ABI) with the CPU checkers.

Tolerance: fp64 rel 1e-10, fp32 rel 1e-5 of the tensor's max magnitude (util.relerr)."""
import os
import numpy as np
import pytest
import torch

import util
from ai2pot_b200 import capi, synth

pytestmark = pytest.mark.gpu
G = np.load(os.path.join(util.GOLDEN, "golden_small.npz"))
TOL = {np.float64: 1e-10, np.float32: 1e-5}


def _chk(checkers):
    return checkers.get("ref") or checkers["oracle"]


def _run(w, nb, virial=True):
    dt = torch.float64 if nb["brcs"].dtype == np.float64 else torch.float32
    prog = capi.MtpProgram(w["model"]["tables"])
    md = capi.to_device({k: v for k, v in w["model"].items() if k != "tables"}, float_dtype=dt)
    nbd = capi.to_device(nb)
    out = capi.mtp_efv(prog, md, nbd, virial=virial)
    torch.cuda.synchronize()
    return [o.cpu().numpy() for o in out], prog, md, nbd


def test_g0_golden_and_checker(checkers):
    w = synth.g0(util.tables(10))
    chk = _chk(checkers)
    nb = util.nblist_batch(chk, w)
    (e, f, v), prog, md, nbd = _run(w, nb)
    for a, k in ((e, "g0_e"), (f, "g0_f"), (v, "g0_v")):
        assert util.relerr(a, G[k]) < 1e-10, k
    e2, f2 = capi.mtp_efv(prog, md, nbd, virial=False)
    assert util.relerr(e2.cpu().numpy(), G["g0_e"]) < 1e-10 and util.relerr(f2.cpu().numpy(), G["g0_f"]) < 1e-10
    d = capi.mtp_descriptors(prog, md, nbd).cpu().numpy()
    assert util.relerr(d[0, :8], G["g0_desc_head"]) < 1e-10
    assert util.relerr(d, chk.mtp_descriptors(w["model"], nb)) < 1e-10


@pytest.mark.parametrize("level,dt", [(6, np.float64), (16, np.float64), (10, np.float32)])
def test_small_golden(checkers, level, dt):
    w = util.small_mtp_case(level, 5, dt)
    nb = util.nblist_batch(_chk(checkers), w)
    (e, f, v), *_ = _run(w, nb)
    tag = f"mtp{level}_{np.dtype(dt).name}"
    for a, k in ((e, "_e"), (f, "_f"), (v, "_v")):
        assert util.relerr(a, G[tag + k]) < TOL[dt], k


def test_g1_slice_vs_checker(checkers):
    """Level 16 / rcut 6 (the benchmark model) on a 12^3 lattice against the CPU checker."""
    w = synth.g1(util.tables(16), n=12)
    chk = _chk(checkers)
    nb = util.nblist_batch(chk, w)
    (e, f, v), *_ = _run(w, nb)
    er, fr, vr = chk.mtp_efv(w["model"], nb)
    assert util.relerr(e, er) < 1e-10 and util.relerr(f, fr) < 1e-10 and util.relerr(v, vr) < 1e-10


def test_g1_full_size_vs_checker(checkers):
    """configs[1] itself: level 16, fp64, 13,824 atoms, rcut 6 - energy, forces and virial against the CPU code at
    rel 1e-10 (neighbour list from the CPU code; the CUDA list is compared bit for bit in test_nblist_gpu.py)."""
    w = synth.g1(util.tables(16))
    chk = _chk(checkers)
    nb = util.nblist_batch(chk, w)
    (e, f, v), *_ = _run(w, nb)
    er, fr, vr = chk.mtp_efv(w["model"], nb)
    errs = dict(energy=util.relerr(e, er), force=util.relerr(f, fr), virial=util.relerr(v, vr))
    print("configs[1] full size, CUDA vs CPU code:", errs)
    assert max(errs.values()) < 1e-10, errs


@pytest.mark.parametrize("natoms,level,dt", [(3, 16, np.float64), (133, 16, np.float32), (1777, 16, np.float64), (2370, 10, np.float64), (3001, 10, np.float32),
                                             (5003, 10, np.float64), (9001, 10, np.float32), (15001, 6, np.float64)])
def test_lanes_share_the_slots_of_an_atom(checkers, natoms, level, dt):
    """Structures of a size for 8, 4, 2 and 1 lanes per atom, contraction tiles of 16 and 32 atoms, blocks of 32 and 8 warps, the last tile ragged, some
    atoms at an open side with few neighbours; fp32 against the model in double precision (every input is a single)."""
    rng = np.random.default_rng(natoms)
    edge = int(np.ceil(natoms ** (1 / 3) - 1e-9))
    cell, pos = synth.cubic_lattice(max(edge, 4), 3.0, 0.1, rng, np.float64, nocc=natoms)
    w = util.small_mtp_case(level, 2, dt)
    w.update(cell=cell, coords=pos.astype(dt).astype(np.float64), types=rng.integers(0, 3, natoms).astype(np.int32))
    chk = _chk(checkers)
    nb = util.nblist_batch(chk, w)
    if dt == np.float32:
        nb["brcs"] = nb["brcs"].astype(dt)
    (e, f, v), *_ = _run(w, nb)
    model = util.to64(w["model"])
    er, fr, vr = chk.mtp_efv(model, dict(nb, brcs=nb["brcs"].astype(np.float64)))
    for a, r, name in ((e, er, "energy"), (f, fr, "force"), (v, vr, "virial")):
        assert util.relerr(a, r) < TOL[dt], name


@pytest.mark.parametrize("natoms", [7201, 14211])
def test_a_lane_per_atom_in_single_precision(checkers, natoms):
    """Level 16, fp32: the force kernel of full tiles (first size), and the one of shared slots right beyond a round of full tiles; with and without
    virial. Against the model in double precision; four times the distance of the CPU code's own single-precision result."""
    rng = np.random.default_rng(natoms)
    cell, pos = synth.cubic_lattice(int(np.ceil(natoms ** (1 / 3) - 1e-9)), 3.0, 0.1, rng, np.float64, nocc=natoms)
    w = util.small_mtp_case(16, 2, np.float32)
    w.update(cell=cell, coords=pos.astype(np.float32).astype(np.float64), types=rng.integers(0, 3, natoms).astype(np.int32))
    chk = _chk(checkers)
    nb = util.nblist_batch(chk, w)
    nb["brcs"] = nb["brcs"].astype(np.float32)
    (e, f, v), prog, md, nbd = _run(w, nb)
    e2, f2 = capi.mtp_efv(prog, md, nbd, virial=False)
    ref = chk.mtp_efv(util.to64(w["model"]), dict(nb, brcs=nb["brcs"].astype(np.float64)))
    tol = [max(TOL[np.float32], 4 * util.relerr(o, r)) for o, r in zip(chk.mtp_efv(w["model"], nb), ref)]
    for a, k, name in ((e, 0, "energy"), (f, 1, "force"), (v, 2, "virial"), (e2.cpu().numpy(), 0, "energy"), (f2.cpu().numpy(), 1, "force")):
        assert util.relerr(a, ref[k]) < tol[k], name


@pytest.mark.parametrize("natoms", [27, 2400])
def test_tables_that_fit_tiles_of_32_atoms_only(checkers, natoms):
    """Sixteen moments in a chain, each the sum of 300 products: the rows of a tile of 16 atoms (four groups of lanes per warp, of
    which one moment fills one) take twice the shared memory of those of 32, more than the tile itself saves."""
    levels, rows = 16, 300
    rng = np.random.default_rng(natoms)
    tables = dict(alpha_moments_count=4 + levels, nmus=1, alpha_moment_mapping=np.arange(4 + levels, dtype=np.int32),
                  alpha_index_basic=np.array([[0, 0, 0, 0], [0, 1, 0, 0], [0, 0, 1, 0], [0, 0, 0, 1]], np.int32),
                  alpha_index_times=np.array([(3 + k if k else 0, r % 4, 1, 4 + k) for k in range(levels) for r in range(rows)], np.int32))
    cell, pos = synth.cubic_lattice(int(np.ceil(natoms ** (1 / 3) - 1e-9)), 3.0, 0.1, rng, np.float64, nocc=natoms)
    w = dict(cell=cell, coords=pos, types=rng.integers(0, 3, natoms).astype(np.int32), rcut=5.0, umax=48,
             model=synth.mtp_model(tables, 3, rng, np.float64, 5.0, 0.5, sigma=0.1))
    chk = _chk(checkers)
    nb = util.nblist_batch(chk, w)
    desc = chk.mtp_descriptors(w["model"], nb)
    w["model"].update(q_scaler=np.abs(desc[0]).max(0), linear_coeffs=rng.normal(0, 1, desc.shape[2]))      # every scalar counts
    (e, f, v), prog, md, nbd = _run(w, nb)
    e2, f2 = capi.mtp_efv(prog, md, nbd, virial=False)
    er, fr, vr = chk.mtp_efv(w["model"], nb)
    for a, r, name in ((e, er, "energy"), (f, fr, "force"), (v, vr, "virial"), (e2.cpu().numpy(), er, "energy"), (f2.cpu().numpy(), fr, "force"),
                       (capi.mtp_descriptors(prog, md, nbd).cpu().numpy(), desc, "descriptors")):
        assert util.relerr(a, r) < 1e-10, name


@pytest.mark.parametrize("level,dt,natoms", [(6, np.float64, 5003), (10, np.float64, 4737), (10, np.float32, 9001)])
def test_blocks_of_eight_warps_without_virial(checkers, level, dt, natoms):
    """Small tables with more tiles than SMs: energy and forces without the virial, and descriptors."""
    rng = np.random.default_rng(natoms)
    cell, pos = synth.cubic_lattice(int(np.ceil(natoms ** (1 / 3) - 1e-9)), 3.0, 0.1, rng, np.float64, nocc=natoms)
    w = util.small_mtp_case(level, 2, dt)
    w.update(cell=cell, coords=pos.astype(dt).astype(np.float64), types=rng.integers(0, 3, natoms).astype(np.int32))
    chk = _chk(checkers)
    nb = util.nblist_batch(chk, w)
    nb["brcs"] = nb["brcs"].astype(dt)
    model, nb64 = util.to64(w["model"]), dict(nb, brcs=nb["brcs"].astype(np.float64))
    (e, f), prog, md, nbd = _run(w, nb, virial=False)
    er, fr, _ = chk.mtp_efv(model, nb64)
    for a, r, name in ((e, er, "energy"), (f, fr, "force"), (capi.mtp_descriptors(prog, md, nbd).cpu().numpy(), chk.mtp_descriptors(model, nb64), "descriptors")):
        assert util.relerr(a, r) < TOL[dt], name


@pytest.mark.parametrize("nm,nt,kmu,dt", [(110, 64, (4, 2, 0), np.float64), (230, 100, (6, 4, 2, 0), np.float64), (230, 100, (6, 4, 2, 0), np.float32)])
def test_few_products_over_many_moments(checkers, nm, nt, kmu, dt):
    """Few products, more tiles than SMs: blocks of 32 warps where three of eight do not fit an SM (the second case). Single precision:
    four times the distance of the CPU code's own single-precision result."""
    natoms = 5003
    rng = np.random.default_rng(nm)
    cell, pos = synth.cubic_lattice(int(np.ceil(natoms ** (1 / 3) - 1e-9)), 3.0, 0.1, rng, np.float64, nocc=natoms)
    model = synth.mtp_model(util.synthetic_tables(nm, nt, kmu=kmu), 3, rng, np.float64, 5.0, 0.5, sigma=0.1)
    w = dict(cell=cell, coords=pos.astype(dt).astype(np.float64), types=rng.integers(0, 3, natoms).astype(np.int32), rcut=5.0, umax=48, model=model)
    chk = _chk(checkers)
    nb = util.nblist_batch(chk, w)
    desc = chk.mtp_descriptors(model, nb)
    model.update(q_scaler=np.abs(desc[0]).max(0), linear_coeffs=rng.normal(0, 1, desc.shape[2]))      # every scalar counts
    w["model"] = {k: (v.astype(dt) if isinstance(v, np.ndarray) and v.dtype == np.float64 else v) for k, v in model.items()}
    nb["brcs"] = nb["brcs"].astype(dt)
    got, *_ = _run(w, nb)
    ref = chk.mtp_efv(util.to64(w["model"]), dict(nb, brcs=nb["brcs"].astype(np.float64)))
    own = ref if dt == np.float64 else chk.mtp_efv(w["model"], nb)
    for a, r, o, name in zip(got, ref, own, ("energy", "force", "virial")):
        assert util.relerr(a, r) < max(TOL[dt], 4 * util.relerr(o, r)), name


def test_many_neighbours_and_ragged_batch(checkers):
    """> 32 neighbours per atom (two lane chunks), padded batch with an empty structure and ghosts."""
    chk = _chk(checkers)
    rng = np.random.default_rng(3)
    lists, mxs = [], []
    for n, a in ((4, 2.2), (3, 2.5), (5, 2.0)):
        cell, pos = synth.cubic_lattice(n, a, 0.1, rng)
        ty = rng.integers(0, 2, len(pos)).astype(np.int32)
        nn, fn, rc, _, mx = chk.nblist(cell, ty, pos, 4.8, 128)
        mxs.append(mx)
        lists.append((nn, fn, rc, ty))
    assert max(mxs) > 64 and min(mxs) < 32      # one, two and three lane chunks
    nb = synth.pad_batch(lists, 2, 128)
    nb["binum"][1] = 0                     # an empty structure in the middle of the batch
    model = synth.mtp_model(util.tables(10), 2, rng, np.float64, 4.8, 1.0)
    w = dict(model=model)
    (e, f, v), *_ = _run(w, nb)
    er, fr, vr = chk.mtp_efv(model, nb)
    assert e[1] == 0 and np.all(f[1] == 0)
    assert util.relerr(e, er) < 1e-10 and util.relerr(f, fr) < 1e-10 and util.relerr(v, vr) < 1e-10


def test_properties_full_size():
    """Size-independent checks at the benchmark size (13,824 atoms, level 16) with a GPU-free
    neighbour list: net force zero, symmetric virial, invariance under atom relabelling."""
    from oracle import refapi
    w = synth.g1(util.tables(16))
    chk = refapi.Checker("oracle")
    nb = util.nblist_batch(chk, w)
    (e, f, v), prog, md, nbd = _run(w, nb)
    fs = np.abs(f).max()
    assert np.abs(f[0].sum(0)).max() < 1e-9 * fs * len(f[0])
    V = v.reshape(3, 3)
    assert np.abs(V - V.T).max() < 1e-9 * np.abs(V).max()
    # second run is bit-for-bit repeatable in energy up to atomic ordering
    e2, f2, v2 = capi.mtp_efv(prog, md, nbd)
    assert util.relerr(e2.cpu().numpy(), e) < 1e-12 and util.relerr(f2.cpu().numpy(), f) < 1e-12
    # outputs are overwritten, whatever they held (the set-up launch zeroes them: there are no memsets)
    dirty = tuple(torch.full_like(x, float("nan")) for x in (e2, f2, v2))
    e3, f3, v3 = capi.mtp_efv(prog, md, nbd, out=dirty)
    assert util.relerr(e3.cpu().numpy(), e) < 1e-12 and util.relerr(f3.cpu().numpy(), f) < 1e-12
    assert util.relerr(v3.cpu().numpy(), v) < 1e-12


def test_errors():
    t = util.tables(10)
    bad = dict(t)
    bad["alpha_index_basic"] = t["alpha_index_basic"].copy()
    bad["alpha_index_basic"][3, 1] = 12    # degree beyond the supported maximum
    with pytest.raises(capi.Ai2bError):
        capi.MtpProgram(bad)
    # host tensors are refused: there is no CPU path behind the C ABI
    w = util.small_mtp_case(6, 3)
    from oracle import refapi
    nb = util.nblist_batch(refapi.Checker("oracle"), w)
    nb_host = {k: (torch.from_numpy(v) if isinstance(v, np.ndarray) else v) for k, v in nb.items()}
    md = capi.to_device({k: v for k, v in w["model"].items() if k != "tables"})
    with pytest.raises(capi.Ai2bError):
        capi.mtp_efv(capi.MtpProgram(w["model"]["tables"]), md, nb_host)
