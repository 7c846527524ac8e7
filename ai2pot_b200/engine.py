"""Host-side driver of the evaluation path: positions -> neighbour list -> E/F/V on one GPU.
Everything on the device goes through the C ABI."""
import ctypes as C

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
        self.lists = capi.NeighborBuilder.new_outputs(n, self.umax, dtype, dev)     # numneigh, firstneigh, rcs, status
        self.nb_static = dict(binum=torch.tensor([n], dtype=torch.int32, device=dev),
                              bilist=torch.arange(n, dtype=torch.int32, device=dev)[None].contiguous(),
                              btypes=torch.from_numpy(np.ascontiguousarray(types, np.int32)).to(dev)[None].contiguous(),
                              ntypes=int(model["ntypes"]), nghost=0)
        # E, virial and forces in one piece, [E | virial (9) | pad | forces (3 n)], so that a host reads them with one copy
        self.outbuf = torch.empty(16 + 3 * n, dtype=dtype, device=dev)
        self.out = (self.outbuf[0:1], self.outbuf[16:].view(1, n, 3), self.outbuf[1:10].view(1, 9))
        self.status = self.lists[3]
        self.graph = self.graph_io = None
        self._describe()

    def _describe(self):
        """Everything a call needs but the positions, once (ai2b_evaluation)."""
        m, is64 = self.model, self.dtype == torch.float64
        self.nb_ws = torch.empty(max(256, capi.lib().ai2b_nblist_workspace_bytes(C.c_int(self.n), C.c_int(int(is64)))), dtype=torch.uint8, device=self.device)
        if self.kind == "mtp":
            need = capi.lib().ai2b_mtp_workspace_bytes(self.prog.handle, C.c_int(1), C.c_int(self.n), C.c_int(int(m["ntypes"])))
        else:
            need = capi.lib().ai2b_nep_workspace_bytes(C.c_int(1), C.c_int(int(m["ntypes"])), C.c_int(int(m["n_radial"])), C.c_int(int(m["n_angular"])),
                                                       C.c_int(int(m["chebyshev_size"])), C.c_int(int(is64)))
        self.ws = torch.empty(max(need, 256), dtype=torch.uint8, device=self.device)
        d = capi.Evaluation()
        d.is_f64, d.natoms, d.umax, d.ntypes, d.rcut = int(is64), self.n, self.umax, int(m["ntypes"]), self.rcut
        cell = np.asarray(self.cell, np.float64 if is64 else np.float32).reshape(9)
        for k in range(9):
            d.cell[k] = float(cell[k])
        d.chebyshev_size = int(m["chebyshev_size"])
        ptr = lambda t: t.data_ptr()
        if self.kind == "mtp":
            d.mtp, d.scaling, d.rmax, d.rmin, d.d_linear_coeffs = self.prog.handle.value, float(m["scaling"]), float(m["rmax"]), float(m["rmin"]), ptr(m["linear_coeffs"])
        else:
            d.n_radial, d.n_angular, d.l_max, d.num_neurons = (int(m[k]) for k in ("n_radial", "n_angular", "l_max", "num_neurons"))
            d.rmax, d.rmax_angular = float(m["rmax_radial"]), float(m["rmax_angular"])
            d.d_w0, d.d_b0, d.d_w1 = ptr(m["w0"]), ptr(m["b0"]), ptr(m["w1"])
        d.d_coeffs, d.d_type_bias, d.d_q_scaler = ptr(m["coeffs"]), ptr(m["type_bias"]), ptr(m["q_scaler"])
        d.d_binum, d.d_ilist, d.d_types = (ptr(self.nb_static[k]) for k in ("binum", "bilist", "btypes"))
        d.d_numneigh, d.d_firstneigh, d.d_rcs, d.d_status = (ptr(t) for t in self.lists)
        d.d_etot, d.d_force, d.d_virial = (ptr(t) for t in self.out)
        d.d_nblist_workspace, d.nblist_workspace_bytes = ptr(self.nb_ws), self.nb_ws.numel()
        d.d_workspace, d.workspace_bytes = ptr(self.ws), self.ws.numel()
        self._desc, self._call = d, (capi.lib().ai2b_evaluate, C.byref(d), self.device.index)

    def build_list(self, coords):
        nn, fn, rcs, status = self.builder.build(self.cell, coords, self.rcut, self.umax, out=self.lists)
        return dict(self.nb_static, bnumneigh=nn[None], bfirstneigh=fn[None], brcs=rcs[None])

    def evaluate(self, nb):
        if self.kind == "mtp":
            return capi.mtp_efv(self.prog, self.model, nb, out=self.out)
        return capi.nep_efv(self.model, nb, out=self.out, ws=self.ws)

    def compute(self, coords):
        if coords.dtype is not self.dtype or coords.shape[0] != self.n or not coords.is_cuda or not coords.is_contiguous():
            return self.evaluate(self.build_list(coords))
        fn, desc, dev = self._call
        rc = fn(desc, coords.data_ptr(), capi.raw_stream(dev))
        if rc:
            capi._check(rc)
        return self.out

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
            self.graph = g
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
        try:
            torch.cuda.synchronize()
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g):
                capi.copy_around_call(coords, host_coords)
                self.compute(coords)
                capi.copy_around_call(host_out, self.outbuf)
            self.graph_io = g
        except Exception:
            self.graph_io = None
            torch.cuda.synchronize()
        return self.graph_io is not None

    def replay_io(self):
        self.graph_io.replay()

    # kernels of this library launched by one compute() on a fully periodic cell (memsets not counted): neighbour build =
    # binning (one launch up to 2,048 atoms, else set-up, count, fill, with a scan between them for many bins) and rows;
    # MTP = forward, contraction, force (plus a set-up launch when the radial coefficient rows have to be padded to eight
    # entries); NEP = zeroing of the outputs + one kernel
    def launches_per_step(self):
        bins = 1
        for d in self.cell_heights():
            bins *= max(1, int(d / (self.rcut * 1.0001 + 1e-6)))
        build = 2 if self.n <= 2048 else 4 if bins <= 8192 else 5
        if self.kind == "mtp":
            return build + 3 + (0 if int(self.model["chebyshev_size"]) == 8 else 1)
        return build + 2

    def cell_heights(self):
        """Distances between opposite faces of the cell."""
        c = self.cell.astype(np.float64)
        return abs(np.linalg.det(c)) / np.array([np.linalg.norm(np.cross(c[(k + 1) % 3], c[(k + 2) % 3])) for k in range(3)])
