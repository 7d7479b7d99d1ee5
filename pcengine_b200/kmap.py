"""Host-side kernel-map object: owns the device arrays the C ABI fills and
derives the other forms lazily.  Mirrors what the reference keeps per
(kernel size, tensor stride, layer stride) in ``spTensor.kmaps``
(script/spconv.py:333,382-384,431-433)."""
from __future__ import annotations

import ctypes as C
from typing import Optional, Sequence

import torch

from . import _lib
from ._lib import lib

D1_CODE = 1186111  # backend/hash.cuh:7-9


def make_geom(ks, stride, pad, cmin, cmax, subm: bool) -> _lib.Geom:
    g = _lib.Geom()
    for i in range(3):
        g.ks[i] = int(ks[i])
        g.stride[i] = int(stride[i])
        g.pad[i] = int(pad[i])
        g.cmin[i] = int(cmin[i])
        g.cmax[i] = int(cmax[i])
    g.submanifold = 1 if subm else 0
    return g


def candidates_per_input(ks, stride) -> int:
    """Upper bound on the outputs one input voxel can feed in a strided conv."""
    n = 1
    for k, s in zip(ks, stride):
        n *= (k + s - 1) // s
    return n


def leads_to_parents(ks, stride, pad, subm: bool) -> bool:
    """Whether a layer's outputs are the parents of its inputs, through at most 32 offsets."""
    return not subm and tuple(ks) == tuple(stride) and not any(pad) and ks[0] * ks[1] * ks[2] <= 32


# Rows per tile of the tile lists (128 or 256) when the caller does not say.
TILE_ROWS = 128


class NeighbourCSR:
    """mask [rows, ceil(kv/32)] uint32 (as int32 storage), rowptr [rows+1], nbr [cap].

    What the convolutions read may be another form than rowptr / nbr, which are then built on first use by ``fill``, a
    callable returning (rowptr, nbr):

    * ``lists`` (starts, nbr): a row's neighbours from nbr[starts[row]] on (starts None: entry ``row``), as
      pce_subm_neighbours leaves them;
    * ``table``: the dense [kv, rows] table of this direction (a map of at most 32 offsets); the mask then appears with
      the row order, or with rowptr / nbr (``mask_ready`` False until then);
    * neither: a planned map whose tile lists were filled by the planner.

    ``counts``: device int32 [kv], rows that have each offset.
    ``parents``: a direction of a map between voxels and their parents (:func:`leads_to_parents`)."""

    __slots__ = ("_mask", "_rowptr", "_nbr", "n_rows", "n_src", "kv", "_order", "_tiles", "_fp32", "_fill", "_pairs", "_lists",
                 "_table", "_counts", "_mask_ready", "parents")

    def __init__(self, mask, rowptr, nbr, n_rows, n_src, kv=None, fill=None, pairs=None, lists=None, table=None, counts=None,
                 mask_ready=True, parents=False):
        self._mask, self._rowptr, self._nbr, self.n_rows, self.n_src = mask, rowptr, nbr, n_rows, n_src
        self.kv = kv
        self._order = None
        self._tiles = {}
        self._fp32 = None
        self._fill = fill
        self._pairs = pairs  # callable -> one-element device tensor, for a CSR without rowptr
        self._lists, self._table, self._counts, self._mask_ready = lists, table, counts, mask_ready
        self.parents = parents

    def pair_count(self) -> torch.Tensor:
        """Number of (row, offset) pairs as a NEW one-element device tensor (no read-back, and nothing that
        keeps the map's storage alive)."""
        if self._rowptr is None and self._pairs is not None:
            return self._pairs()
        return self.rowptr[-1:].clone()

    def _materialise(self):
        if self._rowptr is None and self._fill is not None:
            self._rowptr, self._nbr = self._fill()
            self._mask_ready = True  # (a fill that is given an empty mask writes it)
            self._fill = None

    @property
    def mask(self):
        if not self._mask_ready:
            self._materialise()
        return self._mask

    @property
    def rowptr(self):
        self._materialise()
        return self._rowptr

    @property
    def nbr(self):
        self._materialise()
        return self._nbr

    def row_lists(self):
        """(starts, nbr): every row's first neighbour and the neighbours, in whatever form is at hand."""
        if self._rowptr is None and self._lists is not None and self._lists[0] is not None:
            return self._lists
        return self.rowptr, self.nbr

    def restrict(self, n_rows: int) -> "NeighbourCSR":
        """The CSR of the first ``n_rows`` output rows only (same inputs, shared storage): what a
        slab of a scene uses to compute its owned rows and not the halo's."""
        if not 0 <= n_rows <= self.n_rows:
            raise ValueError("restrict: n_rows out of range")
        if self._rowptr is None and self._lists is not None and self._lists[0] is not None:
            starts, nbr = self._lists
            return NeighbourCSR(self.mask[:max(n_rows, 1)], None, None, n_rows, self.n_src, self.kv, lists=(starts[: max(n_rows, 1)], nbr),
                                fill=lambda: (self.rowptr[: n_rows + 1], self.nbr),
                                pairs=lambda: self.rowptr[n_rows: n_rows + 1].clone(), parents=self.parents)
        return NeighbourCSR(self.mask[:max(n_rows, 1)], self.rowptr[: n_rows + 1], self.nbr, n_rows, self.n_src, self.kv,
                            parents=self.parents)

    def order(self):
        """Output rows sorted by indicator bitmask (int32 [n_rows], built once): the order in which
        the tensor-core kernel forms its 128-row tiles."""
        if self._order is None and self.n_rows == 0:
            self._order = torch.empty((0,), dtype=torch.int32, device=self._mask.device)
        if self._order is None and self.kv is not None:
            dev = self._mask.device
            out = torch.empty((self.n_rows,), dtype=torch.int32, device=dev)
            ws = _lib.workspace(64 * self.n_rows + (16 << 20), dev)
            _lib.check(lib.pce_csr_sort_rows_counted(self.mask.data_ptr(), _lib.ptr(self._counts), self.n_rows, self.kv,
                                                     ws.data_ptr(), ws.numel(), out.data_ptr(), _lib.stream_ptr(dev)),
                       "pce_csr_sort_rows_counted")
            self._order = out
        return self._order

    def lists_fp32(self):
        """The lists of the tiled fp32 kernel (sorted rows, 128 per tile, one offset per stage), built on first use.
        Kept apart from ``tiles``, which feed the tensor cores."""
        hit = self._fp32
        if hit is None:
            hit = self._fp32 = self._build_tiles(True, 128, False, 1)
        return hit[0]

    def tiles(self, sort_rows: bool = True, tile_rows: int | None = None, identity: bool = False, slots: int = 1):
        """The map as tile lists (a ``_lib.TileLists`` struct of device pointers) for the
        tensor-core kernel; built once per CSR, ordering, tile height and ``identity`` (every tile
        ends with the stage where a second operand joins) and ``slots`` (offsets per stage: 64 / C_in
        for layers with 16 or 32 input channels), kept alive with it.  A request without ``identity``
        is also served by lists that have the stage: the kernel skips it."""
        tile_rows = int(tile_rows or TILE_ROWS)
        key = (bool(sort_rows), tile_rows, bool(identity), int(slots))
        hit = self._tiles.get(key)
        if hit is None and not identity:
            hit = self._tiles.get((bool(sort_rows), tile_rows, True, int(slots)))
        if hit is None:
            hit = self._tiles[key] = self._build_tiles(*key)
        return hit[0]

    def _build_tiles(self, sort_rows: bool, tile_rows: int, identity: bool, slots: int):
        dev = self._mask.device
        n_tiles = (self.n_rows + tile_rows - 1) // tile_rows
        cap = max(1, n_tiles * ((self.kv + slots - 1) // slots + (1 if identity else 0)))
        hit = _TileSet(cap * slots, tile_rows, n_tiles, dev)
        tile_ptr, stage_kp, stage_nbr = hit.pointers()
        if sort_rows and self._order is None and self.kv <= 32 and self.n_rows > 0:
            order = self._order_and_lists(tile_rows, identity, slots, tile_ptr, stage_kp, stage_nbr, cap)
        else:
            order = self.order() if sort_rows else torch.arange(self.n_rows, dtype=torch.int32, device=dev)
            starts, nbr = self.row_lists()
            ws = _lib.workspace(8 * (n_tiles + 1) + (1 << 20), dev)
            _lib.check(lib.pce_build_tile_lists(self.mask.data_ptr(), starts.data_ptr(), nbr.data_ptr(), order.data_ptr(),
                                                self.n_rows, self.kv, tile_rows, 1 if identity else 0, int(slots), ws.data_ptr(),
                                                ws.numel(), tile_ptr, stage_kp, stage_nbr, cap,
                                                _lib.stream_ptr(dev)), "pce_build_tile_lists")
        hit.order = order
        hit.struct = _lib.TileLists(order.data_ptr(), tile_ptr, stage_kp, stage_nbr, tile_rows, 1 if identity else 0, int(slots), 0)
        return hit

    def _order_and_lists(self, tile_rows, identity, slots, tile_ptr, stage_kp, stage_nbr, cap):
        """The row order (kept) and one set of lists in one launch, from the form at hand."""
        dev = self._mask.device
        order = torch.empty((self.n_rows,), dtype=torch.int32, device=dev)
        starts = nbr = table = None
        if self._rowptr is None and self._lists is not None:
            starts, nbr = self._lists
        elif self._rowptr is None and self._table is not None:
            table = self._table
        else:
            starts, nbr = self.rowptr, self.nbr
        want = _lib.TileLists(order.data_ptr(), tile_ptr, stage_kp, stage_nbr, tile_rows, 1 if identity else 0, int(slots), 0)
        caps = (C.c_int32 * 1)(cap)
        ws = _lib.workspace(lib.pce_order_workspace_bytes(self.n_rows), dev)
        _lib.check(lib.pce_order_lists(self._mask.data_ptr(), _lib.ptr(starts), _lib.ptr(nbr), _lib.ptr(table),
                                       _lib.ptr(self._counts), self.n_rows, self.kv, order.data_ptr(), C.byref(want), caps, 1,
                                       ws.data_ptr(), ws.numel(), _lib.stream_ptr(dev)), "pce_order_lists")
        self._order = order
        if table is not None:
            self._mask_ready = True
        return order


class _TileSet:
    """One set of tile lists: (struct, order, tile_ptr, stage_kp, stage_nbr), the lists in one allocation, whose parts
    become tensors when somebody asks."""

    __slots__ = ("struct", "order", "store", "parts")

    def __init__(self, entries: int, tile_rows: int, n_tiles: int, device):
        self.parts = (entries * tile_rows, entries, n_tiles + 1)
        self.store = torch.empty((sum(self.parts),), dtype=torch.int32, device=device)

    def pointers(self):
        at = self.store.data_ptr()
        return at + 4 * (self.parts[0] + self.parts[1]), at + 4 * self.parts[0], at

    def __getitem__(self, i):
        nbr, kp, ptr = self.store.split_with_sizes(self.parts) if i != 0 else (None, None, None)
        return (self.struct, self.order, ptr, kp, nbr)[i]


class _DenseTables:
    """The dense map of a layer, map[kv][n_in] and (unless the map is its own transpose) map_out[kv][n_out], with its
    per-offset counts: built on first use.  An object of its own, so that what derives from it later (a CSR's rowptr and
    nbr) does not have to hold the KernelMap that holds the CSR."""

    NAMES = ("map", "map_out", "knnz", "kpos", "qkpos", "status")

    def __init__(self, in_coords, out_coords, geom, kv, mid, subm, symmetric):
        self.in_coords, self.out_coords, self.geom, self.kv, self.mid = in_coords, out_coords, geom, kv, mid
        self.subm, self.symmetric = subm, symmetric
        self.n_in, self.n_out = int(in_coords.size(0)), int(out_coords.size(0))
        self.built = False

    def build(self) -> "_DenseTables":
        """Hash the output coordinates, query every (input, offset) and scan the per-offset counts
        (idempotent), on PyTorch's current stream."""
        if self.built:
            return self
        dev, kv, in_coords = self.in_coords.device, self.kv, self.in_coords
        st = _lib.stream_ptr(dev)
        ws = _lib.workspace(lib.pce_map_workspace_bytes(self.n_in, kv, self.n_out), dev)
        self.map = torch.empty((kv * self.n_in,), dtype=torch.int32, device=dev)
        # A submanifold map with odd kernel sizes is its own transpose under kp -> kv-1-kp, so
        # the output-major table is read out of `map`; otherwise it is written separately.
        self.map_out = None if self.symmetric else torch.empty((kv * max(self.n_out, 1),), dtype=torch.int32, device=dev)
        # one array, so that one copy reads the totals back: [knnz | kpos | qkpos | status]
        self.words = torch.zeros((3 * kv + 3,), dtype=torch.int32, device=dev)
        self.knnz, self.kpos, self.qkpos, self.status = self.words.split_with_sizes((kv, kv + 1, kv + 1, 1))
        _lib.check(lib.pce_map_build_d2(in_coords.data_ptr(), self.n_in, self.out_coords.data_ptr(), self.n_out,
                                        C.byref(self.geom), ws.data_ptr(), ws.numel(), _lib.ptr(self.map),
                                        self.knnz.data_ptr(), self.kpos.data_ptr(), self.qkpos.data_ptr(),
                                        _lib.ptr(self.map_out), self.status.data_ptr(), st), "pce_map_build_d2")
        self.built = True
        return self

    def csr(self, transposed: bool, pairs: Optional[int] = None):
        """(mask, rowptr, nbr) of one direction; ``pairs``: their number, when known."""
        self.build()
        dev, kv = self.in_coords.device, self.kv
        st = _lib.stream_ptr(dev)
        ident = self.mid if self.subm else -1
        if self.symmetric:
            # the table read with kp reversed is the output-major one; under `transposed`
            # (roles swapped) the table itself is.
            table, n_rows, reverse = self.map, self.n_out, (0 if transposed else 1)
        elif transposed:
            table, n_rows, reverse = self.map, self.n_in, 0
        else:
            table, n_rows, reverse = self.map_out, self.n_out, 0
        words = (kv + 31) // 32
        cap = max(1, kv * min(self.n_in, self.n_out) if not self.subm else kv * self.n_in)
        if pairs is not None:
            cap = max(1, pairs + (self.n_in if self.subm else 0))
        mask = torch.empty((max(n_rows, 1), words), dtype=torch.int32, device=dev)
        rowptr = torch.empty((n_rows + 1,), dtype=torch.int32, device=dev)
        nbr = torch.empty((cap,), dtype=torch.int32, device=dev)
        ws = _lib.workspace(8 * (n_rows + 1) + (8 << 20), dev)
        _lib.check(lib.pce_csr_from_dense(_lib.ptr(table), kv, n_rows, reverse, ident, ws.data_ptr(), ws.numel(),
                                          mask.data_ptr(), rowptr.data_ptr(), nbr.data_ptr(), cap, st),
                   "pce_csr_from_dense")
        return mask, rowptr, nbr


class KernelMap:
    def __init__(self, in_coords: torch.Tensor, ks, stride, pad, cmin, cmax_out, subm: bool):
        _lib.require_cuda(in_coords, "coords")
        if in_coords.dtype != torch.int32 or in_coords.dim() != 2 or in_coords.size(1) != 4:
            raise ValueError("coords must be an int32 [N,4] tensor of (b,x,y,z)")
        in_coords = _lib.whole_rows(in_coords)
        dev = in_coords.device
        self.device = dev
        self.ks, self.stride, self.pad = tuple(ks), tuple(stride), tuple(pad)
        self.subm = bool(subm)
        self.kv = int(ks[0] * ks[1] * ks[2])
        self.mid = (ks[0] - 1) // 2 * ks[1] * ks[2] + (ks[1] - 1) // 2 * ks[2] + (ks[2] - 1) // 2
        self.n_in = int(in_coords.size(0))
        self.in_coords = in_coords
        self.geom = make_geom(ks, stride, pad, cmin, cmax_out, subm)
        st = _lib.stream_ptr(dev)
        kv = self.kv
        # The block form (kmap_blocks.cu): submanifold maps with odd sizes up to 5, and layers whose outputs are the
        # parents of their inputs; it leaves what the convolutions read, and the dense table is built when asked for.
        self._blocks = bool(subm) and all(k % 2 == 1 and k <= 5 for k in ks) and 1 < kv <= 128
        self._parents = None
        if subm:
            self.out_coords = in_coords
            self.n_out = self.n_in
        elif not self._build_parents(st):
            cap = max(1, self.n_in * candidates_per_input(ks, stride))
            ws = _lib.workspace(lib.pce_map_workspace_bytes(self.n_in, kv, cap), dev)
            oc = torch.empty((cap, 4), dtype=torch.int32, device=dev)
            n_out = C.c_int32(0)
            _lib.check(lib.pce_downsample_coords(in_coords.data_ptr(), self.n_in, C.byref(self.geom), ws.data_ptr(),
                                                 ws.numel(), oc.data_ptr(), cap, C.byref(n_out), st),
                       "pce_downsample_coords")
            self.n_out = int(n_out.value)
            self.out_coords = oc[: self.n_out]
        self._csr: dict = {}
        self._pairs = None
        self._d1 = None
        self._sizes = None
        self._state = None
        self.dataflow = "D2"
        # A submanifold map with odd kernel sizes is its own transpose under kp -> kv-1-kp, so
        # the output-major table is read out of `map`; otherwise it is written separately.
        self.symmetric = self.subm and all(k % 2 == 1 for k in ks)
        self._dense = _DenseTables(in_coords, self.out_coords, self.geom, kv, self.mid, self.subm, self.symmetric)
        if not self._blocks and self._parents is None:
            self.build()

    def __getattr__(self, name):
        if name in _DenseTables.NAMES and "_dense" in self.__dict__:
            return getattr(self._dense.build(), name)
        raise AttributeError(name)

    def _build_parents(self, st) -> bool:
        """The map between the inputs and their parents (kernel size == stride, no padding): output coordinates and
        both directions at once.  False when the layer, or a very sparse cloud, needs the general form."""
        ks, dev, kv, n = self.ks, self.device, self.kv, self.n_in
        if not leads_to_parents(ks, self.stride, self.pad, self.subm) or n == 0:
            return False
        ws = _lib.workspace(lib.pce_parents_workspace_bytes(n), dev)
        oc = torch.empty((n, 4), dtype=torch.int32, device=dev)
        up_mask = torch.empty((n, 1), dtype=torch.int32, device=dev)
        rows = torch.empty(((kv + 1) * n,), dtype=torch.int32, device=dev)
        up_nbr, child = rows[:n], rows[n:]
        counts = torch.empty((32,), dtype=torch.int32, device=dev)
        n_out = C.c_int32(0)
        status = lib.pce_parents(self.in_coords.data_ptr(), n, C.byref(self.geom), ws.data_ptr(), ws.numel(), oc.data_ptr(),
                                 up_mask.data_ptr(), up_nbr.data_ptr(), child.data_ptr(), counts.data_ptr(), C.byref(n_out), st)
        if status in (_lib.PCE_ERR_TABLE_FULL, _lib.PCE_ERR_UNSUPPORTED):
            return False
        _lib.check(status, "pce_parents")
        self.n_out = int(n_out.value)
        self.out_coords = oc[: self.n_out]
        self._parents = (up_mask, up_nbr, child, counts)
        return True

    def build(self) -> "KernelMap":
        """The dense tables (idempotent), on PyTorch's current stream."""
        self._dense.build()
        return self

    # -- sizes that live on the device -------------------------------------
    def sizes(self):
        """(pairs, qsum) read back once (one synchronisation), also validates the status word.
        The reference reads qkpos[-1] the same way (script/spconv.py:376,421)."""
        if self._sizes is None and self._state is not None and not self._dense.built:
            state = self._state.cpu().tolist()  # rows per offset: a pair per row, the centre apart
            if state[0] != 0:
                _lib.check(state[0], "kernel map build")
            pairs = [v for kp, v in enumerate(state[32: 32 + self.kv]) if kp != self.mid]
            self._sizes = (sum(pairs), sum((v + 127) // 128 * 128 for v in pairs))
        if self._sizes is None:
            host = self._dense.build().words.tolist()
            if host[-1] != 0:
                _lib.check(host[-1], "kernel map build")
            self._sizes = (host[2 * self.kv], host[-2])
        return self._sizes

    # -- neighbour CSR + bitmask (what pce_conv_fwd consumes) ---------------
    def csr(self, transposed: bool = False) -> NeighbourCSR:
        key = bool(transposed)
        if key in self._csr:
            return self._csr[key]
        if self._blocks and not key and not self._dense.built:
            self._csr[key] = self._csr_from_blocks()
            return self._csr[key]
        if self._parents is not None and not self._dense.built:
            self._csr[key] = self._csr_of_parents(key)
            return self._csr[key]
        mask, rowptr, nbr = self._dense.csr(key, self._sizes[0] if self._sizes is not None else None)
        n_rows, n_src = (self.n_in, self.n_out) if key else (self.n_out, self.n_in)
        out = self._csr[key] = NeighbourCSR(mask, rowptr, nbr, n_rows, n_src, self.kv,
                                            parents=leads_to_parents(self.ks, self.stride, self.pad, self.subm))
        return out

    def _csr_from_blocks(self) -> NeighbourCSR:
        dev, kv, n = self.device, self.kv, self.n_in
        words = (kv + 31) // 32
        mask = torch.empty((max(n, 1), words), dtype=torch.int32, device=dev)
        starts = torch.empty((max(n, 1),), dtype=torch.int32, device=dev)
        nbr = torch.empty((max(kv * n, 1),), dtype=torch.int32, device=dev)
        state = torch.empty((160,), dtype=torch.int32, device=dev)
        ws = _lib.workspace(lib.pce_subm_workspace_bytes(n), dev)
        _lib.check(lib.pce_subm_neighbours(self.in_coords.data_ptr(), n, C.byref(self.geom), ws.data_ptr(), ws.numel(),
                                           mask.data_ptr(), starts.data_ptr(), nbr.data_ptr(), state.data_ptr(),
                                           _lib.stream_ptr(dev)), "pce_subm_neighbours")
        self._state = state
        counts, dense = state[32: 32 + kv], self._dense
        return NeighbourCSR(mask, None, None, n, n, kv, fill=lambda: dense.csr(False)[1:], lists=(starts, nbr), counts=counts,
                            pairs=lambda: counts.sum(0, keepdim=True, dtype=torch.int32))

    def _csr_of_parents(self, transposed: bool) -> NeighbourCSR:
        up_mask, up_nbr, child, counts = self._parents
        pairs = lambda: counts.sum(0, keepdim=True, dtype=torch.int32)
        dense = self._dense
        if transposed:
            return NeighbourCSR(up_mask, None, None, self.n_in, self.n_out, self.kv, fill=lambda: dense.csr(True)[1:],
                                pairs=pairs, lists=(None, up_nbr),
                                counts=counts, parents=True)
        mask = torch.empty((max(self.n_out, 1), 1), dtype=torch.int32, device=self.device)

        def fill():
            full, rowptr, nbr = dense.csr(False)
            mask.copy_(full)
            return rowptr, nbr
        return NeighbourCSR(mask, None, None, self.n_out, self.n_in, self.kv, fill=fill, pairs=pairs, table=child, counts=counts,
                            mask_ready=False, parents=True)

    # -- reference forms -----------------------------------------------------
    def pairs(self):
        """(imap, omap) int32 [P], ordered by (kp, in): script/spconv.py:370-372."""
        if self._pairs is None:
            p, _ = self.sizes()
            dev = self.device
            imap = torch.empty((p,), dtype=torch.int32, device=dev)
            omap = torch.empty((p,), dtype=torch.int32, device=dev)
            ws = _lib.workspace(8 * self.kv * max(self.n_in, 1) + (16 << 20), dev)
            _lib.check(lib.pce_map_pairs(_lib.ptr(self.map), self.kv, self.n_in, ws.data_ptr(), ws.numel(),
                                         imap.data_ptr(), omap.data_ptr(), p, _lib.stream_ptr(dev)), "pce_map_pairs")
            self._pairs = (imap, omap)
        return self._pairs

    def d1(self):
        """(imap_coded [P], icsr [n_in+1], omap_coded [P], ocsr [n_out+1]): the CSR-coded
        gather/scatter map of backend/hash.cu:20-255 with canonical positions."""
        if self._d1 is None:
            d = self._dense.build()
            p, _ = self.sizes()
            dev = self.device
            imap_c = torch.empty((max(p, 1),), dtype=torch.int32, device=dev)
            omap_c = torch.empty((max(p, 1),), dtype=torch.int32, device=dev)
            icsr = torch.empty((self.n_in + 1,), dtype=torch.int32, device=dev)
            ocsr = torch.empty((self.n_out + 1,), dtype=torch.int32, device=dev)
            ws = _lib.workspace(4 * self.kv * self.n_in + 4 * (self.n_in + self.n_out) + (1 << 20), dev)
            _lib.check(lib.pce_map_build_d1(_lib.ptr(d.map), _lib.ptr(d.map_out), self.kv, self.n_in, self.n_out,
                                            1 if d.symmetric else 0, d.kpos.data_ptr(), ws.data_ptr(), ws.numel(),
                                            imap_c.data_ptr(), icsr.data_ptr(), omap_c.data_ptr(), ocsr.data_ptr(),
                                            _lib.stream_ptr(dev)), "pce_map_build_d1")
            self._d1 = (imap_c[:p], icsr, omap_c[:p], ocsr)
        return self._d1


def csr_from_pairs(rows: torch.Tensor, nbrs: torch.Tensor, kpos: torch.Tensor, kv: int, n_rows: int,
                   n_src: int, identity_kp: int = -1) -> NeighbourCSR:
    """Neighbour CSR from (kp, in)-ordered pair lists (the only map data the reference's
    conv_fwd_d2_cuda receives, backend/spconv.h:28-40)."""
    dev = rows.device
    n_pairs = int(rows.numel())
    words = (kv + 31) // 32
    cap = max(1, n_pairs + (n_rows if identity_kp >= 0 else 0))
    mask = torch.empty((max(n_rows, 1), words), dtype=torch.int32, device=dev)
    rowptr = torch.empty((n_rows + 1,), dtype=torch.int32, device=dev)
    nbr = torch.empty((cap,), dtype=torch.int32, device=dev)
    ws = _lib.workspace(lib.pce_csr_from_pairs_workspace_bytes(n_pairs, n_rows), dev)
    _lib.check(lib.pce_csr_from_pairs(_lib.ptr(rows), _lib.ptr(nbrs), kpos.data_ptr(), kv, n_pairs, n_rows,
                                      identity_kp, ws.data_ptr(), ws.numel(), mask.data_ptr(), rowptr.data_ptr(),
                                      nbr.data_ptr(), cap, _lib.stream_ptr(dev)), "pce_csr_from_pairs")
    return NeighbourCSR(mask, rowptr, nbr, n_rows, n_src, kv)
