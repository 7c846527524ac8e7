"""Drop-in for the reference's CPython module ``nblist`` (source/nblist/bind/nblist_bind.cc:35-207),
backed by the CUDA cell-list builder through the C ABI.

    find_info4mlff(cell, types, coords, rcut, umax, is_cart, pbc, sort)
        -> (inum, ilist, numneigh, firstneigh, rcs, types, nghost)

Same argument order, dtypes (float32 / float64 selected by ``coords``; int64 types are narrowed to
int32) and return tuple as the reference. TypeError on wrong Python types, like the reference;
a row longer than ``umax`` raises (the reference silently overruns its buffer there).
"""
import ctypes as C
import threading

import numpy as np
import torch

from .. import capi

STAGING_BYTES = 64 << 20      # longest list that travels through pinned memory kept between calls
PIECE_BYTES = 8 << 20         # piece of a longer list: two of them are in pinned memory during a call


class _Lists:
    """Device and pinned host buffers for the lists of one size, [status | numneigh | firstneigh | rcs] in one piece, so that
    they come back with a few large transfers. From pageable memory, array by array, the way back was three quarters of a
    call (2,197 atoms, umax 64: 4 MB, 305 of 405 us). Lists above STAGING_BYTES have no host buffers of their own, they
    come back in pieces (262,144 atoms, umax 64: 470 MB, 32 ms; from pageable memory, array by array, 217)."""

    def __init__(self, n, umax, dtype, device):
        self.key = (n, umax, dtype, device)
        self.n, self.umax = n, umax
        size = torch.empty(0, dtype=dtype).element_size()
        up = lambda b: (b + 255) & ~255
        self.at = [0, 256, 256 + up(4 * n), 256 + up(4 * n) + up(4 * n * umax)]
        total = self.at[3] + size * 3 * n * umax
        self.dev = torch.empty(total, dtype=torch.uint8, device=device)
        self.dev[:256].zero_()        # (an empty system's status is not written)
        self.staged = total <= STAGING_BYTES
        self.host = torch.empty(total, dtype=torch.uint8, pin_memory=True) if self.staged else None
        cut = lambda b, k, count, t: b[self.at[k]:self.at[k] + count * torch.empty(0, dtype=t).element_size()].view(t)
        parts = ((0, 2, torch.int32), (1, n, torch.int32), (2, n * umax, torch.int32), (3, 3 * n * umax, dtype))
        self.d = [cut(self.dev, *p) for p in parts]
        self.h = [cut(self.host, *p) for p in parts] if self.staged else None
        self.coords = torch.empty(3 * n, dtype=dtype, device=device)
        self.h_coords = torch.empty(3 * n, dtype=dtype, pin_memory=True) if self.staged else None
        is64 = dtype == torch.float64
        lib = capi.lib()
        need = lib.ai2b_nblist_workspace_bytes(C.c_int(n), C.c_int(int(is64)))
        self.ws = torch.empty(max(need, 256), dtype=torch.uint8, device=device)
        self.build_fn = lib.ai2b_nblist_build_f64 if is64 else lib.ai2b_nblist_build_f32
        self.sort_fn = lib.ai2b_nblist_sort_rows_f64 if is64 else lib.ai2b_nblist_sort_rows_f32
        p = [C.c_void_p(t.data_ptr()) for t in self.d]
        self.tail = (C.c_int(umax), p[1], p[2], p[3], p[0], C.c_void_p(self.ws.data_ptr()), C.c_size_t(self.ws.numel()))
        self.sort_args = (C.c_int(n), C.c_int(umax), p[1], p[2], p[3])
        self.events = [torch.cuda.Event() for _ in range(3)]

    def run(self, cell, coords, rcut, is_cart, pbc, sort):
        current = torch.cuda.current_stream()
        stream = C.c_void_p(current.cuda_stream)
        if self.staged:
            np.copyto(self.h_coords.numpy(), coords.reshape(-1))
            self.coords.copy_(self.h_coords, non_blocking=True)
        else:
            self.coords.copy_(torch.from_numpy(np.ascontiguousarray(coords).reshape(-1)))
        hpbc = (C.c_int * 3)(*[1 if p else 0 for p in pbc])
        capi._check(self.build_fn(C.c_int(self.n), C.c_void_p(cell.ctypes.data), C.c_void_p(self.coords.data_ptr()), C.c_int(1 if is_cart else 0),
                                  C.c_double(rcut), hpbc, *self.tail, stream))
        if sort:
            capi._check(self.sort_fn(*self.sort_args, stream))
        if not self.staged:
            return self.by_pieces(current)
        # rows come back in three pieces; a piece that has arrived is copied out (by all host threads) while the next one travels
        mid = self.at[3] + (self.host.numel() - self.at[3]) // 512 * 256
        for (a, b), ev in zip(((0, self.at[3]), (self.at[3], mid), (mid, self.host.numel())), self.events):
            self.host[a:b].copy_(self.dev[a:b], non_blocking=True)
            ev.record(current)
        nn, fn = torch.empty(self.n, dtype=torch.int32), torch.empty((self.n, self.umax), dtype=torch.int32)
        rcs = torch.empty((self.n, self.umax, 3), dtype=self.coords.dtype)
        self.events[0].synchronize()
        st = self.h[0].tolist()
        nn.copy_(self.h[1])
        fn.view(-1).copy_(self.h[2])
        flat, half = rcs.view(torch.uint8).view(-1), mid - self.at[3]
        self.events[1].synchronize()
        flat[:half].copy_(self.host[self.at[3]:mid])
        self.events[2].synchronize()
        flat[half:].copy_(self.host[mid:])
        return st, nn.numpy(), fn.numpy(), rcs.numpy()

    def by_pieces(self, stream):
        """The lists in pieces of PIECE_BYTES through two pinned buffers, one being copied out while the other is filled."""
        shapes = ((self.n,), (self.n, self.umax), (self.n, self.umax, 3))
        out = [torch.empty(shape, dtype=d.dtype) for d, shape in zip(self.d[1:], shapes)]
        pieces = []
        for d, h in zip(self.d[1:], out):
            src, dst = d.view(torch.uint8), h.view(-1).view(torch.uint8)
            pieces += [(src[a:a + PIECE_BYTES], dst[a:a + PIECE_BYTES]) for a in range(0, src.numel(), PIECE_BYTES)]
        pinned = [torch.empty(PIECE_BYTES, dtype=torch.uint8, pin_memory=True) for _ in range(2)]
        for k in range(len(pieces) + 1):
            if k < len(pieces):
                src = pieces[k][0]
                pinned[k & 1][:src.numel()].copy_(src, non_blocking=True)
                self.events[k & 1].record(stream)
            if k > 0:
                dst = pieces[k - 1][1]
                self.events[(k - 1) & 1].synchronize()
                dst.copy_(pinned[(k - 1) & 1][:dst.numel()])
        return [self.d[0].tolist()] + [h.numpy() for h in out]


_lock = threading.Lock()
_lists = None      # buffers of the last size, if they are staged (at most STAGING_BYTES); replaced when the size changes


def find_info4mlff(cell, types, coords, rcut, umax, is_cart, pbc, sort):
    global _lists
    if not isinstance(cell, np.ndarray) or not isinstance(types, np.ndarray) or not isinstance(coords, np.ndarray):
        raise TypeError("cell, types and coords must be numpy arrays")
    if not isinstance(pbc, (list, tuple)) or len(pbc) != 3:
        raise TypeError("pbc must be a list of three bools")
    if coords.dtype not in (np.float32, np.float64) or cell.dtype != coords.dtype:
        raise TypeError("cell and coords must both be float32 or both float64")
    if types.dtype not in (np.int32, np.int64):
        raise TypeError("types must be int32 or int64")
    cell = np.ascontiguousarray(cell).reshape(9)      # (a cell of another size raises)
    n, umax = int(coords.shape[0]), int(umax)
    key = (n, umax, torch.float64 if coords.dtype == np.float64 else torch.float32, torch.device("cuda", torch.cuda.current_device()))
    with _lock:
        if _lists is None or _lists.key != key:
            _lists = None
            lists = _Lists(*key)
            _lists = lists if lists.staged else None
        else:
            lists = _lists
        try:
            st, nn, fn, rcs = lists.run(cell, coords, float(rcut), bool(is_cart), pbc, bool(sort))
        except Exception:
            torch.cuda.current_stream().synchronize()      # work may be under way on buffers that another stream is given next
            raise
    if st[1]:
        raise ValueError(f"umax={umax} is smaller than the largest neighbour count {st[0]}")
    return (n, np.arange(n, dtype=np.int32), nn, fn, rcs, np.ascontiguousarray(types, dtype=np.int32), 0)
