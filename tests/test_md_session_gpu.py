"""Device-resident MD input path (ai2b_md_session_*): a periodic system is handed over the way an MD
host holds it (local atoms + ghost images, double positions, model types), and the folded forces,
the energy and the six virial components must equal the periodic evaluation of the checker."""
import numpy as np
import pytest

import util
from ai2pot_b200 import capi, synth

pytestmark = pytest.mark.gpu


def _chk(checkers):
    return checkers.get("ref") or checkers["oracle"]


def _with_ghosts(cell, coords, types, rcut):
    """Local atoms wrapped into an orthorhombic box + images with any coordinate within rcut of it."""
    L = np.diag(cell).astype(np.float64)
    x = np.mod(coords.astype(np.float64), L)
    gx, gt, owner = [], [], []
    for sx in (-1, 0, 1):
        for sy in (-1, 0, 1):
            for sz in (-1, 0, 1):
                if sx == sy == sz == 0:
                    continue
                y = x + np.array([sx, sy, sz]) * L
                keep = np.all((y > -rcut) & (y < L + rcut), axis=1)
                gx.append(y[keep]); gt.append(types[keep]); owner.append(np.nonzero(keep)[0])
    return x, np.concatenate(gx), np.concatenate(gt), np.concatenate(owner)


def _fold(f, nlocal, owner):
    out = f[:nlocal].copy()
    np.add.at(out, owner, f[nlocal:])
    return out


def test_md_session_nep(checkers):
    chk = _chk(checkers)
    w = util.small_nep_case(6, np.float32, a=3.0)                      # 216 atoms, 18 A box, rcut 6
    m = w["model"]
    x, gx, gt, owner = _with_ghosts(w["cell"], w["coords"], w["types"], 6.0)
    nlocal, nghost = len(x), len(gx)
    # periodic reference on the same (wrapped, float-rounded as the host would see them in double) positions
    nb = util.nblist_batch(chk, dict(w, coords=x.astype(np.float64), cell=w["cell"].astype(np.float64), umax=96))
    nb["brcs"] = nb["brcs"].astype(np.float32)
    e_ref, f_ref, v_ref = chk.nep_efv(m, nb)
    ses = capi.MdSession(m, 96)
    for _ in range(2):                                                  # second step reuses every buffer
        e, f, v6, mx = ses.compute(nlocal, nghost, np.concatenate([x, gx]), np.concatenate([w["types"], gt]))
        assert 20 < mx <= 96
        assert abs(e - e_ref[0]) < 1e-5 * abs(e_ref[0])
        assert util.relerr(_fold(f, nlocal, owner), f_ref[0]) < 1e-5
        assert util.relerr(v6, v_ref[0][[0, 4, 8, 1, 2, 5]]) < 1e-5
    # growing the system re-allocates; a too small umax is reported, not overrun
    tight = capi.MdSession(m, 8)
    with pytest.raises(capi.Ai2bError):
        tight.compute(nlocal, nghost, np.concatenate([x, gx]), np.concatenate([w["types"], gt]))
    tight.close(); ses.close()


def test_md_session_mtp(checkers):
    chk = _chk(checkers)
    w = util.small_mtp_case(10, 5, np.float32, rcut=5.0)                # 125 atoms, 15 A box
    m = w["model"]
    x, gx, gt, owner = _with_ghosts(w["cell"], w["coords"], w["types"], 5.0)
    nlocal, nghost = len(x), len(gx)
    nb = util.nblist_batch(chk, dict(w, coords=x.astype(np.float64), cell=w["cell"].astype(np.float64), umax=64))
    nb["brcs"] = nb["brcs"].astype(np.float32)
    e_ref, f_ref, v_ref = chk.mtp_efv(m, nb)
    prog = capi.MtpProgram(m["tables"])
    ses = capi.MdSession(m, 64, prog)
    e, f, v6, mx = ses.compute(nlocal, nghost, np.concatenate([x, gx]), np.concatenate([w["types"], gt]))
    assert abs(e - e_ref[0]) < 1e-5 * max(abs(e_ref[0]), np.abs(f_ref).max())
    assert util.relerr(_fold(f, nlocal, owner), f_ref[0]) < 1e-5
    assert util.relerr(v6, v_ref[0][[0, 4, 8, 1, 2, 5]]) < 1e-5
    e2, f2, _, _ = ses.compute(nlocal, nghost, np.concatenate([x, gx]), np.concatenate([w["types"], gt]), want_virial=False)
    assert util.relerr(_fold(f2, nlocal, owner), f_ref[0]) < 1e-5
    ses.close()


@pytest.mark.parametrize("n", [1, 6143, 6144, 6145, 15797, 15798, 18431, 18432, 18433, 30001])
def test_md_session_pieces(n):
    """Positions go to the device in pieces of 6,144 atoms through a ring of three: sizes around a piece, around what the ring
    holds with the types, and beyond the ring; a smaller and a larger system in between."""
    rng = np.random.default_rng(n)
    m = synth.nep_model(3, rng, rmax_radial=4.0, rmax_angular=3.0)
    edge = int(np.ceil(n ** (1.0 / 3.0)))
    g = np.stack(np.meshgrid(*[np.arange(edge) * 2.5] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    x = np.ascontiguousarray(g + rng.normal(0, 0.1, (n, 3)) - 7.0)
    t = rng.integers(0, 3, n).astype(np.int32)
    nlocal = max(1, n - n // 3)
    ses = capi.MdSession(m, 64)
    want = None
    for k in range(3):
        e, f, v, mx = ses.compute(nlocal, n - nlocal, x, t)
        if k == 0:
            import torch
            rows = capi.NeighborBuilder().build(np.eye(3), torch.from_numpy(x).cuda(), 4.0, 64, pbc=(False,) * 3, ncentres=nlocal)
            md = capi.to_device(m)
            nb = dict(binum=torch.tensor([nlocal], dtype=torch.int32, device="cuda"), bilist=torch.arange(nlocal, dtype=torch.int32, device="cuda")[None],
                      bnumneigh=rows[0][None], bfirstneigh=rows[1][None], brcs=rows[2].float()[None].contiguous(),
                      btypes=torch.from_numpy(t).cuda()[None], ntypes=3, nghost=n - nlocal)
            want = [o.cpu().numpy() for o in capi.nep_efv(md, nb)]
            assert mx == int(rows[3][0])
        assert abs(e - want[0][0]) <= 1e-5 * max(1.0, abs(want[0][0])) and (n == 1 or util.relerr(f, want[1][0]) < 1e-5)
        assert n == 1 or util.relerr(v, want[2][0][[0, 4, 8, 1, 2, 5]]) < 1e-5
        small = max(1, n // 2) if k == 0 else n + n // 2       # the buffers serve the smaller one and grow for the larger one
        y = np.resize(x, (small, 3)) + np.arange(small)[:, None] // n * 1000.0
        ses.compute(small, 0, y, np.resize(t, small))
    ses.close()


@pytest.mark.parametrize("kind", ["nep", "mtp"])
def test_first_step_of_a_session(kind):
    """The first step of a session allocates what later steps use: 0.6 to 0.8 ms on a quiet machine (2.1 to 5 with eight device
    allocations and pinned memory for a whole step). The best of several against 1 ms and what one device allocation of that
    size takes at the time, as other users of the machine make allocations slow."""
    import ctypes as C
    import time
    rt = C.CDLL("libcudart.so.12")

    def allocation():
        p = C.c_void_p()
        t0 = time.perf_counter()
        assert rt.cudaMalloc(C.byref(p), C.c_size_t(24 << 20)) == 0 and rt.cudaFree(p) == 0
        return time.perf_counter() - t0
    w = synth.g2(n=24) if kind == "nep" else util.small_mtp_case(16, 14, np.float32, rcut=6.0)
    m = w["model"]
    prog = capi.MtpProgram(m["tables"]) if kind == "mtp" else None
    x = np.ascontiguousarray(np.mod(w["coords"].astype(np.float64), np.diag(w["cell"]).astype(np.float64)))
    first, plain = [], []
    for _ in range(10):
        ses = capi.MdSession(m, 64, prog)
        t0 = time.perf_counter()
        ses.compute(len(x), 0, x, w["types"])
        first.append(time.perf_counter() - t0)
        ses.close()
        plain.append(allocation())
    assert min(first) < 1e-3 + min(plain)


def test_atom_that_has_flown_off():
    """A local atom at infinity or with an undefined position: nobody's neighbour, all other forces are those without it."""
    rng = np.random.default_rng(2)
    m = synth.nep_model(3, rng)
    x = np.stack(np.meshgrid(*[np.arange(9) * 2.8] * 3, indexing="ij"), -1).reshape(-1, 3) + rng.normal(0, 0.1, (729, 3))
    t = rng.integers(0, 3, 729).astype(np.int32)
    ses = capi.MdSession(m, 96)
    e, f, v, mx = ses.compute(729, 0, x, t)
    lone = ses.compute(1, 0, x[:1], t[:1])[0]
    for bad in ([np.inf, 0, 0], [0, -np.inf, 5.0], [np.nan] * 3, [1e30, 1e30, -1e30]):
        e2, f2, v2, mx2 = ses.compute(730, 0, np.concatenate([[bad], x]), np.concatenate([t[:1], t]))
        assert mx2 == mx and not f2[0].any() and util.relerr(f2[1:], f) < 1e-5
        assert abs(e2 - lone - e) < 1e-5 * abs(e) and util.relerr(v2, v) < 1e-5
    ses.close()
