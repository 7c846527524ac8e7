"""Host-side driver of the evaluation path: positions -> neighbour list -> E/F/V on one GPU.
Everything on the device goes through the C ABI."""
import ctypes as C
from operator import itemgetter

import numpy as np
import torch

from . import capi


class Evaluator:
    """One structure, one model, one GPU: compute(coords) -> (etot[1], force[1,N,3], virial[1,9]).
    Mirrors what the reference's calculators do per call (neighbour list, then predict_efv:
    ai2pot/models/potential_utils.py:217-268), with every step on the device."""

    def __init__(self, model, cell, types, rcut, umax, dtype):
        self.kind = model["kind"]
        self.dtype = dtype
        self.cell = np.asarray(cell)
        self.rcut, self.umax = float(rcut), int(umax)
        n = len(types)
        self.n = n
        dev = torch.device("cuda", torch.cuda.current_device())
        self.model = capi.to_device({k: v for k, v in model.items() if k != "tables"}, dev, dtype)
        self.prog = capi.MtpProgram(model["tables"]) if self.kind == "mtp" else None
        self.device = dev
        self.builder = capi.NeighborBuilder()
        self.lists = ()
        self._new_lists()
        self.nb_static = dict(binum=torch.tensor([n], dtype=torch.int32, device=dev),
                              bilist=torch.arange(n, dtype=torch.int32, device=dev)[None].contiguous(),
                              btypes=torch.from_numpy(np.ascontiguousarray(types, np.int32)).to(dev)[None].contiguous(),
                              ntypes=int(model["ntypes"]), nghost=0)
        # E, virial and forces in one piece, [E | virial (9) | pad | forces (3 n)], so that a host reads them with one copy
        self.outbuf = torch.empty(16 + 3 * n, dtype=dtype, device=dev)
        self.out = (self.outbuf[0:1], self.outbuf[16:].view(1, n, 3), self.outbuf[1:10].view(1, 9))
        self.ws = None
        self.nb_ws = torch.empty(max(256, capi.lib().ai2b_nblist_workspace_bytes(C.c_int(n), C.c_int(int(dtype == torch.float64)))),
                                 dtype=torch.uint8, device=dev)
        self.graph = self.graph_io = None
        self._desc, self._filled = capi.Evaluation(), None
        self._desc_cell = np.frombuffer(self._desc, np.float64, 9, capi.Evaluation.cell.offset).reshape(3, 3)
        self._call = (capi.lib().ai2b_evaluate, C.byref(self._desc), self.device.index)
        self._describe()

    @staticmethod
    def _let_go(tensors):
        """Buffers that are about to be replaced may still be in use on the stream of the last call, which need not be the one
        that they were made on."""
        for t in tensors:
            if t is not None:
                t.record_stream(torch.cuda.current_stream())

    def _new_lists(self):
        """Neighbour tensors for rows of umax slots: numneigh, firstneigh, rcs, status."""
        self._let_go(self.lists)
        self.lists = capi.NeighborBuilder.new_outputs(self.n, int(self.umax), self.dtype, self.device)
        self.status = self.lists[3]
        self._row_width, self._filled = self.umax, None

    def _workspace(self):
        """Scratch of the evaluation, large enough for the model as it is now."""
        m = self.model
        if self.kind == "mtp":
            need = capi.lib().ai2b_mtp_workspace_bytes(self.prog.handle, C.c_int(1), C.c_int(self.n), C.c_int(int(self.nb_static["ntypes"])))
        else:
            need = capi.lib().ai2b_nep_workspace_bytes(C.c_int(1), C.c_int(int(self.nb_static["ntypes"])), C.c_int(int(m["n_radial"])),
                                                       C.c_int(int(m["n_angular"])), C.c_int(int(m["chebyshev_size"])),
                                                       C.c_int(int(self.dtype == torch.float64)))
        if self.ws is None or self.ws.numel() < need:
            self._let_go((self.ws,))
            self.ws, self._filled = torch.empty(max(need, 256), dtype=torch.uint8, device=self.device), None
        return self.ws

    SCALARS = {"mtp": itemgetter("chebyshev_size", "scaling", "rmax", "rmin"),
               "nep": itemgetter("chebyshev_size", "n_radial", "n_angular", "l_max", "num_neurons", "rmax_radial", "rmax_angular")}
    TENSORS = {"mtp": itemgetter("coeffs", "type_bias", "q_scaler", "linear_coeffs"),
               "nep": itemgetter("coeffs", "type_bias", "q_scaler", "w0", "b0", "w1")}
    ATOMS = itemgetter("binum", "bilist", "btypes")

    def _describe(self):
        """The call's arguments but the positions (ai2b_evaluation), from what the attributes hold now: cell, cutoff, row width
        and model may be assigned or edited between calls. They are written only if they differ from the last call's. (Calls
        back to back hide this; one that is waited for takes 45 instead of 41 us at 216 atoms.)"""
        m, nb, kind = self.model, self.nb_static, self.kind
        if self._row_width != self.umax:
            self._new_lists()
        tensors = (*self.TENSORS[kind](m), *Evaluator.ATOMS(nb), *self.out)
        if not all(map(torch.Tensor.is_contiguous, tensors)):
            self._check_tensors(tensors)
        ptrs = list(map(torch.Tensor.data_ptr, tensors))
        values = (kind, self.rcut, self.umax, nb["ntypes"], None if self.prog is None else self.prog.handle.value, self.SCALARS[kind](m), ptrs)
        if values != self._filled:
            self._check_tensors(tensors)
            self._fill(ptrs)
            self._filled = values
        cell = self.cell
        if type(cell) is not np.ndarray or cell.shape != (3, 3):
            cell = np.asarray(cell).reshape(3, 3)
        self._desc_cell[...] = cell

    @staticmethod
    def _check_tensors(tensors):
        for t in tensors:
            capi._ptr(t)       # raises for host memory and strides

    def _fill(self, ptrs):
        m, d = self.model, self._desc
        d.is_f64, d.natoms, d.umax, d.ntypes, d.rcut = int(self.dtype == torch.float64), self.n, int(self.umax), int(self.nb_static["ntypes"]), float(self.rcut)
        d.chebyshev_size = int(m["chebyshev_size"])
        if self.kind == "mtp":
            d.mtp, d.scaling, d.rmax, d.rmin = self.prog.handle.value, float(m["scaling"]), float(m["rmax"]), float(m["rmin"])
            model_ptrs = ("d_coeffs", "d_type_bias", "d_q_scaler", "d_linear_coeffs")
        else:
            d.mtp = None
            d.n_radial, d.n_angular, d.l_max, d.num_neurons = (int(m[k]) for k in ("n_radial", "n_angular", "l_max", "num_neurons"))
            d.rmax, d.rmax_angular = float(m["rmax_radial"]), float(m["rmax_angular"])
            model_ptrs = ("d_coeffs", "d_type_bias", "d_q_scaler", "d_w0", "d_b0", "d_w1")
        names = model_ptrs + ("d_binum", "d_ilist", "d_types", "d_etot", "d_force", "d_virial")
        for name, p in zip(names, ptrs, strict=True):
            setattr(d, name, p)
        d.d_numneigh, d.d_firstneigh, d.d_rcs, d.d_status = (t.data_ptr() for t in self.lists)
        ws = self._workspace()
        d.d_nblist_workspace, d.nblist_workspace_bytes = self.nb_ws.data_ptr(), self.nb_ws.numel()
        d.d_workspace, d.workspace_bytes = ws.data_ptr(), ws.numel()

    def _check_coords(self, coords):
        """Buffers and types of a call are those of the structure: other positions would run over them."""
        if not coords.is_cuda:
            raise capi.Ai2bError("coords must be a CUDA tensor")
        if coords.dtype is not self.dtype or coords.shape[0] != self.n or coords.numel() != 3 * self.n:
            raise capi.Ai2bError(f"coords must be {self.n} positions of type {self.dtype}")

    def build_list(self, coords):
        self._check_coords(coords)
        if self._row_width != self.umax:
            self._new_lists()
        nn, fn, rcs, status = self.builder.build(self.cell, coords, self.rcut, int(self.umax), out=self.lists)
        return dict(self.nb_static, bnumneigh=nn[None], bfirstneigh=fn[None], brcs=rcs[None])

    def evaluate(self, nb):
        if self.kind == "mtp":
            return capi.mtp_efv(self.prog, self.model, nb, out=self.out)
        return capi.nep_efv(self.model, nb, out=self.out, ws=self._workspace())

    def compute(self, coords):
        self._check_coords(coords)
        if not coords.is_contiguous() or self.nb_static["nghost"]:
            return self.evaluate(self.build_list(coords))
        self._describe()
        fn, desc, dev = self._call
        rc = fn(desc, coords.data_ptr(), capi.raw_stream(dev))
        if rc:
            capi._check(rc)
        return self.out

    def _buffers(self):
        """What a recorded call works on besides its positions: kept alive with the recording."""
        return self.lists, self.ws, self.nb_ws, self.out, self.prog, list(self.model.values()), list(self.nb_static.values())

    def capture(self, coords):
        """Records one compute(coords) (neighbour build + E/F/V, every launch stream-ordered on buffers this
        object owns) into a CUDA graph; replay() then re-runs it on whatever `coords` holds at that time.
        Returns False (and leaves the eager path in place) if the capture is refused."""
        self.graph = None
        try:
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                self.compute(coords)                      # sizes every buffer before the capture
            torch.cuda.current_stream().wait_stream(side)
            torch.cuda.synchronize()
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g):
                self.graph_out = self.compute(coords)
            self.graph, self.graph_buffers = g, (coords, self._buffers())
        except Exception:
            self.graph = None
            torch.cuda.synchronize()
        return self.graph is not None

    def replay(self):
        self.graph.replay()
        return self.graph_out

    def capture_io(self, coords, host_coords, host_out):
        """One CUDA graph for a whole call as a host sees it: pinned host positions -> device, neighbour build, E/F/V,
        results -> pinned host buffer `host_out` (laid out like `outbuf`: E, virial 1..9, forces from element 16).
        replay_io() then costs one graph launch. Returns False if the capture is refused."""
        self.graph_io = None
        self._describe()                                  # sizes every buffer before the capture
        try:
            torch.cuda.synchronize()
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g):
                capi.copy_around_call(coords, host_coords)
                self.compute(coords)
                capi.copy_around_call(host_out, self.outbuf)
            self.graph_io, self.graph_io_buffers = g, (coords, host_coords, host_out, self.outbuf, self._buffers())
        except Exception:
            self.graph_io = None
            torch.cuda.synchronize()
        return self.graph_io is not None

    def replay_io(self):
        self.graph_io.replay()

    def launches_per_step(self):
        """Kernels of this library that one compute() on a fully periodic cell launches (memsets not counted): neighbour build,
        then forward, contraction and force of MTP (and a set-up launch when the radial coefficient rows have to be padded to
        eight entries), or those of NEP (whose set-up goes out with a launch of the build: one more where buffers were replaced by ones
        that it shares with the build)."""
        build = capi.nblist_build_launches(self.n, self.cell, self.rcut)
        if self.kind == "mtp":
            return build + 3 + (0 if int(self.model["chebyshev_size"]) == 8 else 1)
        efv = capi.nep_efv_launches(self.model, self.n, self.umax, self.dtype)
        return build + (1 if efv == 2 else efv)

    def cell_heights(self):
        """Distances between opposite faces of the cell."""
        return capi.cell_heights(self.cell)
