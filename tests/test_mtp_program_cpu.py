"""Compilation of the MTP tables (host code; a user pays for it with every new model)."""
import ctypes as C
import os
import subprocess
import time

import numpy as np
import pytest

import util
from ai2pot_b200 import _build, capi


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


@pytest.fixture(scope="module")
def host_tables(tmp_path_factory):
    """The table compiler as a program of its own, its device memory on the host: tables -> the numbers it reports."""
    d = tmp_path_factory.mktemp("tables")
    here = os.path.dirname(os.path.abspath(__file__))
    subprocess.check_call([_build._nvcc(), "-O1", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", _build.CSRC, "-o", str(d / "host"),
                           os.path.join(here, "mtp_tables_host.cu")])

    def run(t, *mode):
        arrays = [np.ascontiguousarray(t[k], np.int32).ravel() for k in ("alpha_index_basic", "alpha_index_times", "alpha_moment_mapping")]
        head = [int(t["alpha_moments_count"]), len(t["alpha_index_basic"]), len(t["alpha_index_times"]), len(t["alpha_moment_mapping"]), int(t["nmus"])]
        np.concatenate([np.array(head, np.int32)] + arrays).tofile(d / "in")
        return [int(v) for v in subprocess.run([str(d / "host"), str(d / "in"), *mode], check=True, capture_output=True, text=True).stdout.split()]

    return run


ANY_TABLES = pytest.mark.parametrize("tables", [util.tables(6), util.tables(10), util.tables(16), util.synthetic_tables(600, 2000),
                                                util.synthetic_tables(64, 96, squares=0.0)], ids=["6", "10", "16", "600x2000", "few_squares"])


@ANY_TABLES
def test_rows_are_read_to_their_ends(host_tables, tables):
    """A kernel that keeps the rows of the tables in shared memory reads the products' rows and the adjoints' rows, all of them and
    nothing behind them: the square of a moment has one adjoint row where twice its multiplier fits eight bits, other products two."""
    r = tables["alpha_index_times"]
    adjoints = 2 * len(r) - int(((r[:, 0] == r[:, 1]) & (2 * r[:, 2] <= 255)).sum())
    fwd0, rev0, fwd1, rev1, walked, room, _ = host_tables(tables)
    assert (fwd0, rev0, fwd1) == (len(r), 0, len(r))
    assert walked == adjoints
    assert rev1 == adjoints <= room


@ANY_TABLES
def test_moments_are_dealt_in_order_of_their_rows(host_tables, tables):
    """The deal of a phase's rows to warps takes the moments with the most rows first, equal ones side by side."""
    assert host_tables(tables)[-1] == 0


@ANY_TABLES
def test_every_adjoint_that_is_read_is_written(host_tables, tables):
    """A product that no other product and no scalar uses has the adjoint zero, and the rows of its operands read it."""
    assert host_tables(tables, "uses") == [0]


def test_idle_moments_are_filled(host_tables):
    """Moments that are neither basic nor a product are zero, and nothing reads what was not written."""
    assert host_tables(util.tables_with_idle_moments(), "uses") == [0]
