"""Neighbour lists from the CUDA builder: bit-exact with the CPU checkers after canonical sort."""
import os
import numpy as np
import pytest
import torch

import util
from ai2pot_b200 import capi, synth
from ai2pot_b200.fromcc import nblist as nblist_mod

pytestmark = pytest.mark.gpu
G = np.load(os.path.join(util.GOLDEN, "golden_small.npz"))


def _chk(checkers):
    return checkers.get("ref") or checkers["oracle"]


def _gpu(cell, types, coords, rcut, umax, is_cart=True, pbc=(1, 1, 1), sort=False):
    out = nblist_mod.find_info4mlff(np.ascontiguousarray(cell, dtype=coords.dtype), np.asarray(types), coords, rcut, umax,
                                    is_cart, [bool(p) for p in pbc], sort)
    inum, ilist, nn, fn, rc, ty, ng = out
    assert inum == len(coords) and ng == 0 and np.array_equal(ilist, np.arange(inum)) and ty.dtype == np.int32
    return nn, fn, rc


def test_mos2_fixture():
    z = np.load(os.path.join(util.GOLDEN, "mos2_fixture.npz"))
    nn, fn, rc = _gpu(z["cell"].astype(np.float32), z["z"], z["frac"].astype(np.float32), 3.2, 16, is_cart=False, pbc=(1, 1, 0))
    assert nn.max() == 12
    util.assert_nblist_equal((nn, fn, rc), (G["mos2_numneigh"], G["mos2_first"], G["mos2_rcs"]))


def test_g0_golden():
    w = synth.g0(util.tables(10))
    nn, fn, rc = _gpu(w["cell"], w["types"].astype(np.int64), w["coords"], w["rcut"], w["umax"])
    assert np.array_equal(nn, G["g0_numneigh"])
    fs, rs = util.canonical_nblist(nn, fn, rc)
    assert np.array_equal(fs, G["g0_first_sorted"]) and np.array_equal(rs.view(np.uint64), G["g0_rcs_sorted"].view(np.uint64))
    # padding convention
    pad = np.arange(fn.shape[1])[None] >= nn[:, None]
    assert np.all(fn[pad] == -1) and np.all(rc[pad] == 0)


@pytest.mark.parametrize("dt", [np.float64, np.float32])
def test_triclinic_unwrapped_open_axes(checkers, dt):
    chk = _chk(checkers)
    rng = np.random.default_rng(5)
    cell = np.array([[7.0, 0.3, 0.1], [1.5, 6.5, 0.2], [-0.7, 0.9, 8.0]]).astype(dt)
    frac = rng.random((60, 3))
    pos = (frac @ cell.astype(np.float64) + rng.normal(0, 3.0, (60, 3))).astype(dt)
    types = rng.integers(0, 2, 60).astype(np.int32)
    for pbc in ((1, 1, 1), (1, 0, 1), (0, 0, 0), (0, 1, 0)):
        a = _gpu(cell, types, pos, 5.5, 160, pbc=pbc)
        b = chk.nblist(cell, types, pos, 5.5, 160, pbc=pbc)
        util.assert_nblist_equal(a, b[:3])
    a = _gpu(cell, types, frac.astype(dt), 5.5, 160, is_cart=False, sort=True)
    b = chk.nblist(cell, types, frac.astype(dt), 5.5, 160, is_cart=False, sort=True)
    util.assert_nblist_equal(a, b[:3])
    # sorted rows: distances ascending
    d = np.sqrt((a[2].astype(np.float64) ** 2).sum(-1))
    for i in range(len(a[0])):
        assert np.all(np.diff(d[i, :a[0][i]]) >= 0)


@pytest.mark.parametrize("dt", [np.float64, np.float32])
def test_atoms_many_periods_outside_the_cell(checkers, dt):
    """Unwrapped trajectories: some atoms sit hundreds of lattice periods away from the cell. Beyond 127 periods
    the builder leaves its packed-wrap form for full integers; both forms must give the reference algorithm's
    list. Checked against the plain-C restatement: the reference's own CPU build overruns its bins on such input."""
    chk = checkers["oracle"]
    rng = np.random.default_rng(17)
    cell = np.array([[7.0, 0.3, 0.1], [1.5, 6.5, 0.2], [-0.7, 0.9, 8.0]])
    frac = rng.random((80, 3))
    types = rng.integers(0, 2, 80).astype(np.int32)
    for far in (100, 400):   # within / beyond the packed range
        k = rng.integers(-far, far + 1, (80, 3))
        k[::3] = 0           # a third of the atoms stay at home
        pos = ((frac + k) @ cell).astype(dt)
        a = _gpu(cell.astype(dt), types, pos, 5.5, 160)
        b = chk.nblist(cell.astype(dt), types, pos, 5.5, 160)
        util.assert_nblist_equal(a, b[:3])
        assert a[0][::3].min() > 0   # (like the reference, only images within the supercell range count: far atoms get none)


def test_tiny_cell_many_images(checkers):
    chk = _chk(checkers)
    rng = np.random.default_rng(9)
    cell = np.eye(3) * 4.0
    pos = rng.random((3, 3)) * 4.0
    a = _gpu(cell, np.array([0, 1, 0]), pos, 6.0, 256)
    b = chk.nblist(cell, [0, 1, 0], pos, 6.0, 256)
    util.assert_nblist_equal(a, b[:3])
    # one atom alone sees only its own images
    a = _gpu(cell, np.array([0]), pos[:1], 6.0, 64)
    b = chk.nblist(cell, [0], pos[:1], 6.0, 64)
    util.assert_nblist_equal(a, b[:3])


@pytest.mark.parametrize("dt", [np.float64, np.float32])
def test_g1_full_size_vs_checker(checkers, dt):
    """13,824 atoms, rcut 6 (the benchmark structure), both float types."""
    w = synth.g1(util.tables(16))
    chk = _chk(checkers)
    pos = w["coords"].astype(dt); cell = w["cell"].astype(dt)
    a = _gpu(cell, w["types"], pos, 6.0, 64)
    b = chk.nblist(cell, w["types"], pos, 6.0, 64)
    util.assert_nblist_equal(a, b[:3])


def test_g4_slice_float(checkers):
    w = synth.g4(ncell=8)
    chk = _chk(checkers)
    a = _gpu(w["cell"], w["types"], w["coords"], 6.0, 32)
    b = chk.nblist(w["cell"], w["types"], w["coords"], 6.0, 32)
    util.assert_nblist_equal(a, b[:3])


def test_overflow_and_errors():
    w = synth.g0(util.tables(10))
    with pytest.raises(ValueError):
        _gpu(w["cell"], w["types"], w["coords"], 5.0, 8)
    with pytest.raises(TypeError):
        nblist_mod.find_info4mlff(w["cell"].tolist(), w["types"], w["coords"], 5.0, 64, True, [True] * 3, False)
    with pytest.raises(TypeError):
        nblist_mod.find_info4mlff(w["cell"], w["types"], w["coords"].astype(np.float32), 5.0, 64, True, [True] * 3, False)
    # device-level status of a truncated build
    nb = capi.NeighborBuilder()
    nn, fn, rc, st = nb.build(w["cell"], torch.from_numpy(w["coords"]).cuda(), 5.0, 8)
    st = st.cpu().numpy()
    assert st[1] == 1 and st[0] == G["g0_numneigh"].max() and nn.max().item() == 8


def test_empty_structure():
    nb = capi.NeighborBuilder()
    nn, fn, rc, st = nb.build(np.eye(3) * 5, torch.zeros(0, 3, dtype=torch.float64, device="cuda"), 3.0, 8)
    assert nn.numel() == 0


@pytest.mark.parametrize("dt", [np.float64, np.float32])
def test_centre_ranges_bin_reuse_and_host_extent(checkers, dt):
    """ai2b_nblist_build_range_*: rows for a range of centres equal the same rows of the full list; a second range
    built from the bins the first call left in the workspace is identical; a host-given extent along an open
    first axis (even a wrong one: atoms outside it share the edge bins) changes nothing."""
    chk = _chk(checkers)
    rng = np.random.default_rng(8)
    cell, pos = synth.cubic_lattice(8, 2.9, 0.12, rng, dt)
    n = len(pos)
    types = np.zeros(n, np.int32)
    tdt = torch.float64 if dt == np.float64 else torch.float32
    dpos = torch.from_numpy(pos).cuda()
    for pbc in ((True, True, True), (False, True, True)):
        ref = chk.nblist(cell, types, pos, 5.0, 64, pbc=[int(p) for p in pbc])
        b = capi.NeighborBuilder()
        c0, c1, c2 = 37, 300, n
        o1 = capi.NeighborBuilder.new_outputs(c1 - c0, 64, tdt, dpos.device)
        o2 = capi.NeighborBuilder.new_outputs(c2 - c1, 64, tdt, dpos.device)
        b.build(cell, dpos, 5.0, 64, pbc=pbc, ncentres=c1, cbegin=c0, out=o1)
        b.build(cell, dpos, 5.0, 64, pbc=pbc, ncentres=c2, cbegin=c1, reuse_bins=True, out=o2)
        for (nn, fn, rc, st), (lo, hi) in ((o1, (c0, c1)), (o2, (c1, c2))):
            assert int(st[1]) == 0
            util.assert_nblist_equal((nn.cpu().numpy(), fn.cpu().numpy(), rc.cpu().numpy()), (ref[0][lo:hi], ref[1][lo:hi], ref[2][lo:hi]))
        if not pbc[0]:
            frac = pos[:, 0].astype(np.float64) / float(cell[0, 0])
            for ext in ((frac.min(), frac.max()), (0.2, 0.7)):
                o3 = capi.NeighborBuilder.new_outputs(n, 64, tdt, dpos.device)
                capi.NeighborBuilder().build(cell, dpos, 5.0, 64, pbc=pbc, out=o3, open_extent=ext)
                util.assert_nblist_equal((o3[0].cpu().numpy(), o3[1].cpu().numpy(), o3[2].cpu().numpy()), ref[:3])


@pytest.mark.parametrize("dt", [np.float64, np.float32])
def test_batched_build_ragged_triclinic_fractional(checkers, dt):
    """ai2b_nblist_build_batch_*: a ragged batch (one empty structure, one cell thinner than the cutoff, triclinic cells,
    fractional input, an open axis) against the CPU code structure by structure; truncation to umax is flagged."""
    chk = _chk(checkers)
    rng = np.random.default_rng(21)
    tdt = torch.float64 if dt == np.float64 else torch.float32
    cells, fracs, ns = [], [], [40, 0, 9, 75, 130]
    for k, n in enumerate(ns):
        L = (3.4 if k == 2 else 9.0) + k
        cell = (np.eye(3) * L + rng.normal(0, 0.4, (3, 3))).astype(dt)
        cells.append(cell)
        fracs.append((rng.random((n, 3)) * 1.6 - 0.3).astype(dt))          # some atoms outside the cell
    npad = max(ns)
    B = len(ns)
    coords = np.zeros((B, npad, 3), dt)
    for b in range(B):
        coords[b, :ns[b]] = fracs[b]
    for pbc in ((True, True, True), (True, False, True)):
        out = capi.nblist_build_batch(np.stack(cells), torch.tensor(ns, dtype=torch.int32).cuda(), torch.from_numpy(coords).cuda(), 4.5, 200,
                                      is_cart=False, pbc=pbc)
        st = out["status"].cpu().numpy()
        assert st[1] == 0
        mxs = [0]
        for b in range(B):
            n = ns[b]
            if n == 0:
                assert int(out["bnumneigh"][b].abs().sum()) == 0
                continue
            nn, fn, rc, ty, mx = chk.nblist(cells[b], np.zeros(n, np.int32), fracs[b], 4.5, 200, is_cart=False, pbc=[int(p) for p in pbc])
            mxs.append(mx)
            util.assert_nblist_equal((out["bnumneigh"][b, :n].cpu().numpy(), out["bfirstneigh"][b, :n].cpu().numpy(),
                                      out["brcs"][b, :n].cpu().numpy()), (nn, fn, rc))
            assert bool((out["bfirstneigh"][b, n:] == -1).all()) and float(out["brcs"][b, n:].abs().sum()) == 0.0
        assert st[0] == max(mxs)
    small = capi.nblist_build_batch(np.stack(cells), torch.tensor(ns, dtype=torch.int32).cuda(), torch.from_numpy(coords).cuda(), 4.5, 8,
                                    is_cart=False)
    st = small["status"].cpu().numpy()
    assert st[1] & 1 and st[0] > 8 and int(small["bnumneigh"].max()) == 8


@pytest.mark.parametrize("dt", [np.float64, np.float32])
def test_lanes_as_centres_kernel_on_small_cases(checkers, dt, monkeypatch):
    """Large sparse systems take the form with one warp per bin (the test of 1,048,576 atoms runs it at full size).
    AI2B_NBL_MIN_ATOMS = 0 sends every build through it: triclinic cell with atoms outside it, open axes, fractional input, a
    centre range with bin reuse, truncated rows."""
    monkeypatch.setenv("AI2B_NBL_MIN_ATOMS", "0")
    chk = _chk(checkers)
    rng = np.random.default_rng(15)
    cell = np.array([[17.0, 0.3, 0.1], [1.5, 16.5, 0.2], [-0.7, 0.9, 18.0]]).astype(dt)
    frac = rng.random((400, 3))
    pos = (frac @ cell.astype(np.float64) + rng.normal(0, 6.0, (400, 3))).astype(dt)
    types = rng.integers(0, 2, 400).astype(np.int32)
    for pbc in ((1, 1, 1), (1, 0, 1), (0, 0, 0), (0, 1, 0), (1, 1, 0)):
        a = _gpu(cell, types, pos, 5.5, 160, pbc=pbc)
        b = chk.nblist(cell, types, pos, 5.5, 160, pbc=pbc)
        util.assert_nblist_equal(a, b[:3])
    a = _gpu(cell, types, frac.astype(dt), 5.5, 160, is_cart=False)
    b = chk.nblist(cell, types, frac.astype(dt), 5.5, 160, is_cart=False)
    util.assert_nblist_equal(a, b[:3])
    # the benchmark structure, a centre range and bin reuse
    w = synth.g1(util.tables(16))
    p1 = w["coords"].astype(dt); c1 = w["cell"].astype(dt)
    ref = chk.nblist(c1, w["types"], p1, 6.0, 64)
    util.assert_nblist_equal(_gpu(c1, w["types"], p1, 6.0, 64), ref[:3])
    tdt = torch.float64 if dt == np.float64 else torch.float32
    dpos = torch.from_numpy(p1).cuda()
    nb = capi.NeighborBuilder()
    lo, mid, hi = 1000, 5000, 9000
    o1 = capi.NeighborBuilder.new_outputs(mid - lo, 64, tdt, dpos.device)
    o2 = capi.NeighborBuilder.new_outputs(hi - mid, 64, tdt, dpos.device)
    nb.build(c1, dpos, 6.0, 64, ncentres=mid, cbegin=lo, out=o1)
    nb.build(c1, dpos, 6.0, 64, ncentres=hi, cbegin=mid, reuse_bins=True, out=o2)
    for (nn, fn, rc, st), (x0, x1) in ((o1, (lo, mid)), (o2, (mid, hi))):
        util.assert_nblist_equal((nn.cpu().numpy(), fn.cpu().numpy(), rc.cpu().numpy()), (ref[0][x0:x1], ref[1][x0:x1], ref[2][x0:x1]))
    # truncated rows are flagged, the counts are the true ones
    nn, fn, rc, st = capi.NeighborBuilder().build(c1, dpos, 6.0, 8)
    st = st.cpu().numpy()
    assert st[1] == 1 and st[0] == ref[0].max() and nn.max().item() == 8


@pytest.mark.parametrize("dt", [np.float64, np.float32])
@pytest.mark.parametrize("n,density,umax,pbc", [
    (1, 0.03, 64, (1, 1, 1)),
    (37, 0.03, 100, (1, 1, 1)),          # cell narrower than the cutoff: candidates come in pieces
    (2048, 0.03, 64, (1, 1, 1)),         # last size that one block bins
    (2049, 0.03, 63, (1, 1, 1)),         # first size that is binned by several launches; rows without 16-byte alignment
    (2048, 0.03, 64, (0, 1, 0)),
    (2500, 0.03, 64, (0, 0, 0)),         # extents looked up by a cluster of blocks
    (8100, 0.005, 32, (1, 1, 1)),        # sparse bins: two warps per bin
    (8100, 0.0015, 32, (1, 1, 1)),       # ... one warp per bin
    (8100, 0.14, 256, (1, 1, 1)),        # crowded bins: more candidates than the table holds
])
def test_build_at_the_edges_of_its_forms(checkers, dt, n, density, umax, pbc):
    chk = _chk(checkers)
    rng = np.random.default_rng(n)
    L = (n / density) ** (1.0 / 3.0)
    cell = (np.eye(3) * L + np.array([[0, 0, 0], [0.1, 0, 0], [0.05, -0.1, 0]]) * L).astype(dt)
    pos = (rng.random((n, 3)) @ cell.astype(np.float64) + rng.normal(0, 0.3, (n, 3))).astype(dt)
    types = np.zeros(n, np.int32)
    rcut = 5.0 if density < 0.1 else 4.0
    a = _gpu(cell, types, pos, rcut, umax, pbc=pbc)
    b = chk.nblist(cell, types, pos, rcut, umax, pbc=pbc)
    util.assert_nblist_equal(a, b[:3])


@pytest.mark.parametrize("dt", [np.float64, np.float32])
def test_host_list_keeps_no_large_buffers(checkers, dt, monkeypatch):
    """A host list above the staging limit comes back in pieces, and nothing of it stays behind."""
    from ai2pot_b200.fromcc import nblist
    chk = _chk(checkers)
    w = util.small_mtp_case(10, 6, dt)
    args = (w["cell"], w["types"], w["coords"], 5.0, 48, True, [True, True, True])
    ref = chk.nblist(w["cell"], w["types"], w["coords"], 5.0, 48)
    staged = nblist.find_info4mlff(*args, True)
    held = nblist._lists
    assert held is not None and held.host.is_pinned() and held.host.numel() <= nblist.STAGING_BYTES
    monkeypatch.setattr(nblist, "STAGING_BYTES", held.host.numel() - 1)
    monkeypatch.setattr(nblist, "_lists", None)
    for piece in (8 << 20, 4096, 1000 * dt(0).itemsize):
        monkeypatch.setattr(nblist, "PIECE_BYTES", piece)
        plain = nblist.find_info4mlff(*args, True)
        assert nblist._lists is None
        for a, b in zip(plain, staged):
            assert np.array_equal(a, b) and (np.isscalar(a) or a.dtype == b.dtype and a.shape == b.shape and a.flags.writeable)
    util.assert_nblist_equal(nblist.find_info4mlff(*args, False)[2:5], ref[:3])
    monkeypatch.setattr(nblist, "STAGING_BYTES", 1000)
    with pytest.raises(ValueError, match="umax=8"):
        nblist.find_info4mlff(*args[:4], 8, *args[5:], False)
    empty = nblist.find_info4mlff(w["cell"], w["types"][:0], w["coords"][:0], 5.0, 48, True, [True] * 3, True)
    assert empty[0] == 0 and empty[3].shape == (0, 48) and empty[4].shape == (0, 48, 3)


@pytest.mark.parametrize("dt", [np.float64, np.float32])
@pytest.mark.parametrize("n,spacing,form", [(300, 3.0, ""), (3000, 3.0, ""), (9000, 3.0, ""), (9000, 4.2, ""), (9000, 5.5, ""), (3000, 3.0, "0")])
@pytest.mark.parametrize("pbc", [(1, 1, 1), (0, 1, 0)])
def test_atoms_that_have_flown_off(dt, n, spacing, form, pbc, monkeypatch):
    """Infinite, undefined and enormous coordinates: such an atom has no neighbours, and the rows of all others are those of
    the system without it (every form of the row kernel; the bad atoms lie in bins with others)."""
    if form:
        monkeypatch.setenv("AI2B_NBL_MIN_ATOMS", form)
    rng = np.random.default_rng(n)
    edge = int(np.ceil(n ** (1 / 3) - 1e-9))
    cell, pos = synth.cubic_lattice(edge, spacing, 0.1, rng, dt, nocc=n)
    types = np.zeros(n, np.int32)
    want = _gpu(cell, types, pos, 5.0, 64, pbc=pbc)
    far = 1e25 if dt == np.float32 else 1e30
    values = [np.inf, -np.inf, np.nan, far, -far] + ([1e13, -1e13] if dt == np.float64 else [])
    for v in values:
        bad = pos[[0, 1, n // 2]].copy()
        bad[0, 0], bad[1, 1], bad[2] = v, v, v
        nn, fn, rc = _gpu(cell, np.zeros(n + 3, np.int32), np.concatenate([bad, pos]), 5.0, 64, pbc=pbc)
        assert not nn[:3].any() and (fn[:3] == -1).all()
        fn = np.where(fn >= 0, fn - 3, fn)
        assert fn.min() >= -1
        util.assert_nblist_equal((nn[3:], fn[3:], rc[3:]), want)


def test_host_list_that_fails_leaves_no_work_behind(checkers):
    """The buffers of a call that raises half-way (rows too wide to be sorted) may be given to another stream at once."""
    from ai2pot_b200.fromcc import nblist
    w = util.small_mtp_case(10, 6, np.float64)
    args = (w["cell"], w["types"], w["coords"], 5.0, 1500, True, [True, True, True])
    nblist.find_info4mlff(*args, False)         # buffers of this size are there (an allocation would wait for the device)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(100_000_000)          # tens of milliseconds in front of the call's work
        with pytest.raises(capi.Ai2bError):
            nblist.find_info4mlff(*args, True)
        assert side.query()
    ref = _chk(checkers).nblist(w["cell"], w["types"], w["coords"], 5.0, 1500)
    util.assert_nblist_equal(nblist.find_info4mlff(*args, False)[2:5], ref[:3])


@pytest.mark.parametrize("dt", [np.float64, np.float32])
def test_two_warps_per_bin_with_uneven_bins(checkers, dt):
    """Two teams share a block in the two-warp form. Drops in an otherwise empty cell make them run different numbers of bins
    (most are empty) and tables of different length (crowded bins take several pieces), so each needs barriers of its own."""
    chk = _chk(checkers)
    rng = np.random.default_rng(33)
    n, L, rcut, nb = 9000, 70.0, 5.0, 13           # 2,197 bins, 4.1 atoms per bin on average
    drops = rng.random((60, 3)) * L
    sizes = rng.choice([20, 60, 150, 370], size=60)
    pos = np.concatenate([d + rng.normal(0, 2.6, (k, 3)) for d, k in zip(drops, sizes)] + [rng.random((n, 3)) * L])[:n].astype(dt)
    cell, types = (np.eye(3) * L).astype(dt), np.zeros(n, np.int32)
    ref = chk.nblist(cell, types, pos, rcut, 400)
    bins = np.bincount(np.ravel_multi_index((np.floor(np.mod(pos, L) / L * nb).astype(int) % nb).T, (nb, nb, nb)), minlength=nb ** 3)
    assert 2.5 < n / nb ** 3 < 5.5 and (bins == 0).sum() > 500 and bins.max() > 100
    for _ in range(3):
        util.assert_nblist_equal(_gpu(cell, types, pos, rcut, 400), ref[:3])


@pytest.mark.parametrize("dt", [np.float64, np.float32])
@pytest.mark.parametrize("sizes,umax", [((600, 512, 1), 64), ((17, 16, 15), 66)])
def test_batched_build_tiles_and_chunks(checkers, dt, sizes, umax):
    """Structures longer than one tile of the batched build, exactly one tile, and sizes around its chunk of centres."""
    chk = _chk(checkers)
    rng = np.random.default_rng(4)
    B, npad = len(sizes), max(sizes)
    cells = np.stack([np.eye(3) * 3.0 * max(2.0, n ** (1.0 / 3.0)) for n in sizes]).astype(dt)
    coords = np.zeros((B, npad, 3), dt)
    for b, n in enumerate(sizes):
        coords[b, :n] = rng.random((n, 3)) * cells[b, 0, 0]
    out = capi.nblist_build_batch(cells, torch.tensor(sizes, dtype=torch.int32).cuda(), torch.from_numpy(coords).cuda(), 4.0, umax)
    for b, n in enumerate(sizes):
        nn, fn, rc, ty, mx = chk.nblist(cells[b], np.zeros(n, np.int32), coords[b, :n], 4.0, umax)
        util.assert_nblist_equal((out["bnumneigh"][b, :n].cpu().numpy(), out["bfirstneigh"][b, :n].cpu().numpy(),
                                  out["brcs"][b, :n].cpu().numpy()), (nn, fn, rc))


@pytest.mark.parametrize("dt", [np.float64, np.float32])
def test_batched_build_pre_test(checkers, dt):
    """The single-precision test of the batched build drops no neighbour: a structure far from the origin (first atom of the tile or
    not), more than 32 images, an odd count, and atoms with infinite, undefined or enormous coordinates beside whole ones."""
    chk = _chk(checkers)
    rng = np.random.default_rng(12)
    cells, plain = [], []
    for n, L, shift in ((65, 12.0, 0.0), (65, 12.0, 2500.0), (3, 2.1, 0.0), (130, 15.0, -40.0)):
        cells.append(np.eye(3) * L)
        plain.append(rng.random((n, 3)) * L + shift)
    plain[3][1:] += 37 * cells[3][0]                   # the first atom alone in another period
    cells, plain = np.stack(cells).astype(dt), [p.astype(dt) for p in plain]

    def build(frames):
        npad = max(map(len, frames))
        coords = np.zeros((len(frames), npad, 3), dt)
        for b, p in enumerate(frames):
            coords[b, :len(p)] = p
        out = capi.nblist_build_batch(cells, torch.tensor([len(p) for p in frames], dtype=torch.int32).cuda(), torch.from_numpy(coords).cuda(), 4.0, 128)
        return [tuple(out[k][b, :len(p)].cpu().numpy() for k in ("bnumneigh", "bfirstneigh", "brcs")) for b, p in enumerate(frames)]

    want = build(plain)
    for b, p in enumerate(plain):
        nn, fn, rc, ty, mx = chk.nblist(cells[b], np.zeros(len(p), np.int32), p, 4.0, 128)
        util.assert_nblist_equal(want[b], (nn, fn, rc))
    for v in (np.inf, -np.inf, np.nan, 1e25, -1e25) + ((1e13,) if dt == np.float64 else ()):
        bad = np.array([[v, 1.0, 1.0], [1.0, v, 1.0]], dt)
        for got, w in zip(build([np.concatenate([bad, p]) for p in plain]), want):
            nn, fn, rc = got
            assert all((fn[i] == i).sum() == nn[i] and (fn[i] >= 0).sum() == nn[i] for i in (0, 1))      # its own images at most
            fn = np.where(fn >= 0, fn - 2, fn)
            assert fn[2:].min() >= -1
            util.assert_nblist_equal((nn[2:], fn[2:], rc[2:]), w)
