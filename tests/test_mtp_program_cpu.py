"""Compilation of the MTP tables (host code; a user pays for it with every new model)."""
import ctypes as C
import time

import numpy as np
import pytest

import util
from ai2pot_b200 import capi


def _create(t):
    b, r, m = (np.ascontiguousarray(t[k], np.int32) for k in ("alpha_index_basic", "alpha_index_times", "alpha_moment_mapping"))
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    handle, lib = C.c_void_p(), capi.lib()
    t0 = time.perf_counter()
    rc = lib.ai2b_mtp_program_create(C.c_int(int(t["alpha_moments_count"])), C.c_int(len(b)), p(b), C.c_int(len(r)), p(r), C.c_int(len(m)), p(m),
                                     C.c_int(int(t["nmus"])), C.byref(handle))
    dt = time.perf_counter() - t0
    if rc == 0:
        lib.ai2b_mtp_program_destroy(handle)
    return rc, dt


def test_tables_compile_in_a_fraction_of_a_millisecond():
    """Level 16 (350 moments, 969 rows) in at most 1 ms, its upload (which fails without a GPU) included: it takes 0.2 ms, and
    took 2 ms with lists per moment and a trial of every way to split a phase. The best of many, as hosts are busy."""
    t = util.tables(16)
    best = min(_create(t)[1] for _ in range(150))
    assert best < 1e-3


@pytest.mark.parametrize("row,value,why", [(2, 256, "multiplier"), (2, -1, "multiplier"), (3, 41, "out of range"), (0, -1, "out of range")])
def test_bad_rows_are_refused(row, value, why):
    t = dict(util.tables(10))
    t["alpha_index_times"] = t["alpha_index_times"].copy()
    t["alpha_index_times"][5, row] = value
    rc, _ = _create(t)
    assert rc in (-1, -2) and why in capi.lib().ai2b_last_error_string().decode()
