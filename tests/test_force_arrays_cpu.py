"""Memory of the force arrays that an MD session hands out: an array, or anything that looks into it, is the caller's for as
long as it is held (the session writes the next step's forces elsewhere); memory that was let go of is used again."""
import collections
import gc
import sys

import numpy as np
import pytest
import torch

from ai2pot_b200 import capi

HOLDS = {"array": lambda f: f, "slice": lambda f: f[3:5], "view of a view": lambda f: f[::2][1:].T, "reshape": lambda f: f.reshape(-1)[4:],
         "memoryview": memoryview, "tensor": torch.from_numpy, "base": lambda f: f.base, "numpy of a tensor": lambda f: torch.from_numpy(f)[1:].numpy()}


def _session(monkeypatch):
    """A session's force arrays without a device: its forces are the number of the call."""
    calls = []

    class Lib:
        def ai2b_md_session_forces(self, h, nlocal, nghost, x, t, virial, f, e, v, mx):
            n = nlocal.value + nghost.value
            calls.append(f.value)
            capi.C.memmove(f, np.full(3 * n, float(len(calls))).ctypes.data, 24 * n)
            return 0

        def ai2b_md_session_create_nep(self, *a):
            return 0

        def ai2b_md_session_destroy(self, h):
            return 0

    monkeypatch.setattr(capi, "lib", Lib)
    # an interpreter whose counts of references are others than today's must make no difference
    monkeypatch.setattr(sys, "getrefcount", lambda o: 3)
    model = dict(kind="nep", coeffs=0, w0=0, b0=0, w1=0, type_bias=0, q_scaler=0, chebyshev_size=1, n_radial=1, n_angular=0, l_max=0,
                 num_neurons=1, ntypes=1, rmax_radial=1.0, rmax_angular=1.0)
    return capi.MdSession(model, 4), calls


def _step(ses, n=7):
    return ses.compute(n - 2, 2, np.zeros((n, 3)), np.zeros(n, np.int32))[1]


def _values(held):
    return held.block if isinstance(held, capi._Lease) else held


@pytest.mark.parametrize("hold", HOLDS, ids=str)
def test_held_forces_are_not_written_again(monkeypatch, hold):
    ses, _ = _session(monkeypatch)
    kept = [HOLDS[hold](_step(ses)) for _ in range(5)]
    for k, held in enumerate(kept):
        assert np.all(np.asarray(_values(held)) == k + 1.0)
    ses.close()
    ses = None
    gc.collect()
    for k, held in enumerate(kept):
        assert np.all(np.asarray(_values(held)) == k + 1.0)


def test_forces_let_go_of_are_used_again(monkeypatch):
    ses, calls = _session(monkeypatch)
    f = _step(ses)
    assert f.shape == (7, 3) and f.dtype == np.float64 and f.flags.c_contiguous and f.flags.writeable
    for _ in range(6):
        f = _step(ses)          # two blocks in turn: the one in hand and the one of the step before
    assert len(set(calls)) == 2
    del f
    assert len(ses._spare) == 2
    for _ in range(4):          # more than the pool keeps
        kept = [_step(ses) for _ in range(5)]
        del kept
        assert len(ses._spare) == 2
    g = _step(ses, 9)           # another size takes new memory
    assert g.shape == (9, 3) and np.all(g == len(calls))
    ses.close()
    assert not ses._spare


def test_blocks_of_other_shapes_are_dropped():
    pool = collections.deque(maxlen=2)
    a, b = capi._lease_array(pool, (4, 3)), capi._lease_array(pool, (5, 3))
    block = b.ctypes.data
    del a, b
    a = capi._lease_array(pool, (5, 3))
    assert a.ctypes.data == block and len(pool) == 1
    b = capi._lease_array(pool, (6, 3))
    assert b.shape == (6, 3) and not pool
