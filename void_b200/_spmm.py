"""Host side of the SpMM kernels: packed tile store, work plans and the launch itself.

Every function here ends in a call of the C ABI (include/void_b200.h).  Nothing computes on the
CPU; tensors that are not on a CUDA device are rejected.
"""
import functools
import weakref
from dataclasses import dataclass, field
from typing import Optional

import torch

from . import _lib
from .format import check_indexed

TILE = 32
PANEL = 128
CAPTURED = -1   # launch key of a stream that is being captured; others have their stream's
FLAG_DIRECT_STORES, FLAG_A_STABLE = 2, 4   # bits of void_spmm_args.flags
FLAG_NO_EARLY_A = 1 << 30   # host side only: never set FLAG_A_STABLE (measurements)


@dataclass
class PackedTiles:
    """A in the layout the kernels stream: tiles in tile-row-major order, 1024 elements each, already
    in the tensor cores' core-matrix order, with per-tile column index and scale."""
    tiles: torch.Tensor        # uint8 [nnz * 1024 * element bytes], 1024-byte aligned
    tile_cols: torch.Tensor    # int32 [nnz]
    tile_scales: torch.Tensor  # float32 [nnz]
    row_ptr: torch.Tensor      # int32 [nbr + 1]
    block_indices: torch.Tensor  # int32 [nnz]
    row_scale: torch.Tensor    # float32 [nbr]
    nbr: int
    nbc: int
    nnz: int
    shape: tuple
    kind: int                  # _lib.KIND_*
    terms: int = 1             # packed tiles per stored tile (2 / 3: FP8 tiles stored as sums of E4M3 terms)
    stable: bool = False       # the kernels that wrote the arrays above are known to have finished
    row_order: Optional[torch.Tensor] = None   # int32 [nbr]: tile rows by falling tile count (launches without a plan)
    home: Optional[int] = None                 # the stream the arrays were allocated on, if one and known
    native: object = field(default=None, init=False, repr=False, compare=False)   # the native host path's view of this store (handle())

    def is_stable(self) -> bool:
        """True when no kernel still in flight can be writing this store.  A launch may then read
        the store before it waits for the previous kernel of its stream (flag bit 2 of void_spmm_args)."""
        return self.stable

    @functools.cached_property
    def sms(self) -> int:
        return sm_count(self.tiles.device)

    def new_handle(self):
        """What the native host path launches products of this store from, as its fields are now."""
        return _lib.native().packed_handle(
            self.shape[0], self.shape[1], self.kind, self.terms, self.nnz, self.stable, _lib.status_word(self.tiles.device),
            self.tiles, self.tile_cols, self.tile_scales, self.row_ptr, self.row_scale, self.row_order, self.home)

    def handle(self):
        """The handle the operators use, made once."""
        if self.native is None:
            self.native = self.new_handle()
        return self.native


def pack(values: torch.Tensor, scales: Optional[torch.Tensor], block_rows: torch.Tensor, block_cols: torch.Tensor,
         shape, kind: int, row_ptr=None, block_indices=None, terms: int = 1) -> PackedTiles:
    """Build the packed store of a VOID tensor on its device: void_pack_tiles for the 8-bit kinds, with ``terms`` > 1
    void_pack_tiles_f8_split (FP8 tiles with their scales folded in: every tile as a sum of that many E4M3 tiles relative
    to the largest tile scale of its tile row, which lands in row_scale), void_pack_tiles_fp for fp16 / bf16 / fp32 tiles
    (no scales).  The tile index is built on the way unless it is given; _mark_ready waits for all of it and checks it."""
    _lib.require_cuda(values, block_rows, block_cols)
    M, K = shape
    es = _lib.KIND_ELEM_BYTES[kind]
    if values.dim() != 3 or values.shape[1] != TILE or values.shape[2] != TILE or values.element_size() != es:
        raise _lib.VoidB200Error("void_b200 kernels need 32x32 tiles of %d-byte elements here, got %s %s"
                                 % (es, tuple(values.shape), values.dtype))
    tiles, tile_cols, tile_scales, row_ptr, block_indices, row_scale, row_order, home = _lib.native().pack_store(
        values, scales, block_rows, block_cols, M, K, kind, terms, row_ptr, block_indices)
    return PackedTiles(tiles, tile_cols, tile_scales, row_ptr, block_indices, row_scale, (M + TILE - 1) // TILE,
                       (K + TILE - 1) // TILE, values.shape[0], (M, K), kind, terms, row_order=row_order, home=home)


def pack_f8_split(values: torch.Tensor, scales: Optional[torch.Tensor], block_rows: torch.Tensor,
                  block_cols: torch.Tensor, shape, terms: int) -> PackedTiles:
    """Packed store of FP8 tiles with their scales folded in."""
    return pack(values, scales, block_rows, block_cols, shape, _lib.KIND_F8E4M3, terms=terms)


def _mark_ready(p: PackedTiles) -> PackedTiles:
    # Building a packed store is a one-time set-up step of a tensor (a weight): the host waits here until the
    # store is complete, so that every later launch may read it ahead of its stream order.  Inside a stream
    # capture nothing can be waited for, and the arrays hold nothing before the graph is replayed: a store built
    # there is not stable, is never read early, and serves the one product it was built for (it is not kept).
    # The CTAs that start first take the first work items: with the tile rows sorted by falling tile count the
    # longest rows start earliest and the shortest are left for the CTAs that share an SM with the most others.
    p.row_order, indexed = _lib.native().finish_store(p.row_ptr, p.nbr, p.row_order)
    if indexed is not None:
        check_indexed(indexed, p.nnz)
        p.stable = True
    return p


def allow_group_stores(a, allowed: bool) -> None:
    """Whether products of ``a`` (VOIDTensor, Int8VOIDTensor) may keep its tiles a second time, laid out for groups of tile
    rows (by default they may).  From the third large product on of a tensor whose tile rows share enough block columns (up to
    85 - 90 % sparsity), such a store - as large as the packed tiles and a sixteenth more for 8-bit tiles, at most 4 GB, for up to
    two widths of B - is built behind a product and used once it is complete.  False gives the stores of ``a`` back - those that a
    captured graph reads, with ``a`` itself - and keeps further ones from being built."""
    a._group_stores = bool(allowed)
    d = a.__dict__
    for p in (d.get("_packed_cache"), *d.get("_packed_fp_cache", {}).values()):
        if p is not None:
            _lib.native().packed_grouped(p.handle(), bool(allowed))


def retire(owner, *stores) -> None:
    """Stores of ``owner`` whose place is being taken, and its plans, which go with them: those that a captured graph reads stay as
    long as ``owner`` does, so that a replay reads what it was captured with.  (A graph may read a plan and none of these stores:
    that of a product packed inside its capture, or of another operand type.)"""
    kept = [p for p in stores if p is not None and p.native is not None and _lib.native().packed_captured(p.native)]
    plans = [p for p in list(owner.__dict__.get("_plan_cache", {}).values()) if p.captured]
    if kept or plans:
        owner.__dict__.setdefault("_captured_stores", []).append((kept, plans))


def new_store(owner, p: PackedTiles, *made_from) -> PackedTiles:
    """A store that was just packed for ``owner``, ready to be launched from: it knows what it was made from."""
    p = _mark_ready(p)
    _lib.native().packed_made_from(p.handle(), *made_from)
    if not owner.__dict__.get("_group_stores", True):
        _lib.native().packed_grouped(p.native, False)
    return p


def cached_pack(owner, values, scales, block_rows, block_cols, shape, kind) -> PackedTiles:
    """Packed store cached on the tensor object, rebuilt when its storage or contents change."""
    p = owner.__dict__.get("_packed_cache")
    if p is None or not _lib.native().packed_is_current(p.native, values, scales, block_rows, block_cols, shape):
        old, p = p, new_store(owner, pack(values, scales, block_rows, block_cols, shape, kind), values, scales, block_rows,
                              block_cols)
        if p.stable:
            retire(owner, old)
            owner._packed_cache = p
            owner._plan_cache = {}
    return p


_LIVE_PLANS = weakref.WeakSet()


def reset_plan_scratch(device) -> None:
    """Zero the split-row accumulators and counters of every live plan on ``device``.  A launch that gave up
    (status word set) may have left partial sums behind; the kernels only leave the scratch at zero when
    every split row was finished."""
    dev = torch.device(device)
    for plan in list(_LIVE_PLANS):
        if plan.counters.device == dev:
            for partials, counters in list(plan.scratch.values()):
                counters.zero_()
                if partials is not None:
                    partials.zero_()


@dataclass(eq=False)
class Plan:
    """Work plan of void_plan_segments for one (packed tensor, column chunking, CTA count).  The accumulators and counters of
    split rows belong to one launch at a time, so every stream has its own (``partials`` and ``counters`` are those of the
    stream the plan was built on).  Captured launches share one further set: graphs that hold products of the same tensor are
    to be replayed one after the other."""
    segs: torch.Tensor
    cta_seg_ptr: torch.Tensor
    n_cta: int
    np: int
    n_chunks: int
    n_segs: int
    n_slots: int
    n_counters: int
    partials: Optional[torch.Tensor]
    counters: torch.Tensor
    mode: int
    chunk_tiles: int
    # the tile list whose tiles the segments name: its index, the identity of its coordinates, the shape of A
    row_ptr: Optional[torch.Tensor] = None
    tile_list: object = None
    shape: Optional[tuple] = None
    captured: bool = field(default=False, init=False)   # a graph reads it
    scratch: dict = field(default_factory=dict, init=False, repr=False)   # launch key: (partials, counters)

    def __post_init__(self):
        self.scratch[_lib.native().launch_key(self.counters.device.index)] = self.partials, self.counters

    def serves(self, a, packed: PackedTiles) -> bool:
        """Whether the plan was made for the tile list of ``packed``, the store of ``a`` as it is now: from the same index, or from
        one of the same coordinates (a store that is packed inside a capture has an index of its own)."""
        return self.row_ptr is packed.row_ptr or (
            self.tile_list is not None and self.shape == packed.shape
            and _lib.native().unchanged(self.tile_list, a.block_rows, a.block_cols))

    def native_args(self) -> tuple:
        key = _lib.native().launch_key(self.counters.device.index)
        if key == CAPTURED:
            self.captured = True
        partials, counters = self.scratch.get(key) or self._new_scratch(key)
        return self.segs, self.cta_seg_ptr, self.n_cta, partials, counters, self.np

    def _new_scratch(self, key: int) -> tuple:
        """Zeroed accumulators and counters for the current stream (CAPTURED: for captured launches)."""
        if self.partials is None:
            return None, self.counters
        dev, n = self.counters.device, self.partials.numel()
        if key == CAPTURED:      # filled before the graph can run, and not by the graph: a replay leaves them zero again
            both = _lib.native().zeroed_words(n + self.counters.numel(), dev.index)
        else:
            both = torch.zeros(n + self.counters.numel(), dtype=torch.int32, device=dev)
            for t in (self.segs, self.cta_seg_ptr):
                t.record_stream(torch.cuda.current_stream(dev))
        self.scratch[key] = made = both[:n], both[n:]
        return made

    def options(self, acc_out=None, worker_partials=None) -> tuple:
        """The native product call's options for a launch with this plan."""
        return self.native_args(), acc_out, worker_partials, 0, 0, 0, 0, 0, None, 0, 0, None, True


def default_panels(nbr: int, N: int, sms: int) -> int:
    """Panels per work item the library picks by itself (same rule as the C launcher): two, unless
    that leaves fewer work items than four per SM."""
    panels = (N + PANEL - 1) // PANEL
    np_ = 2 if panels >= 2 else 1
    while np_ > 1 and nbr * ((panels + np_ - 1) // np_) < 4 * sms:
        np_ //= 2
    return np_


def sm_count(device) -> int:
    with torch.cuda.device(device):
        return _lib.load().void_device_sm_count()


def streamk_table(row_ptr: torch.Tensor, nbr: int, nnz: int, n_workers: Optional[int], max_work: int):
    """Worker table on the device (void_streamk_table).  Returns the four arrays trimmed to the
    realised worker count, the per-row worker offsets and the chunk length."""
    lib = _lib.load()
    dev = row_ptr.device
    req = -1 if n_workers is None else int(n_workers)
    if nnz == 0 or (n_workers is not None and req <= 0):
        raise ZeroDivisionError("integer division or modulo by zero")  # as void/stream_k.py:66
    target = lib.void_streamk_target(nnz, req, max_work)
    with torch.cuda.device(dev):
        cap = lib.void_streamk_table_capacity(nnz, nbr)
        rows = torch.empty(cap, dtype=torch.int32, device=dev)
        start = torch.empty(cap, dtype=torch.int32, device=dev)
        end = torch.empty(cap, dtype=torch.int32, device=dev)
        atomic = torch.empty(cap, dtype=torch.uint8, device=dev)
        n_out = torch.zeros(1, dtype=torch.int32, device=dev)
        woff = torch.empty(nbr + 1, dtype=torch.int32, device=dev)
        _lib.check(lib.void_streamk_table(_lib.ptr(row_ptr), nbr, nnz, req, max_work, _lib.ptr(rows), _lib.ptr(start),
                                          _lib.ptr(end), _lib.ptr(atomic), _lib.ptr(n_out), _lib.ptr(woff),
                                          _lib.stream_ptr(dev)), "void_streamk_table")
        n = int(n_out.item())
    return rows[:n], start[:n], end[:n], atomic[:n].to(torch.bool), woff, target


ROW_COST = 8   # epilogue of one (tile row, chunk) in units of one tile of work, swept on B200 (power-law rows, N = 256 / 1024, us: 4 15.6 / 45.7, 6 14.4 / 39.4, 8 13.9 / 37.0, 12 14.0 / 37.4, 16 14.8 / 39.4; with contiguous shares: dealt plans take it for whole rows as it is, and four of it for a piece)


def split_mode(nbr: int, n_chunks: int, n_cta: int) -> int:
    """How heavy tile rows are split (split_rows of void_plan_segments): the segments dealt out by weight (3) as long as one
    block can sort them in shared memory, else contiguous shares (1).  Dealt ones were the faster at every size measured below
    that line (27 from 2048 x 2048 to 56000 x 4096; contiguous and dealt, us: 10 - 28 % up to 1300 segments, 30000 x 3000, N = 60 10.7 8.7;
    4096 segments 56.8 51.7, 6400 67.9 61.3 and 56.6 55.5, 7000 61.4 56.9, 5500 of shorter rows 43.7 43.5), so what lies beyond it is
    left for want of room, not because shares even out there."""
    return 3 if n_cta <= 1024 and nbr * n_chunks + 2 * n_cta + 2 <= 8192 else 1


def make_plan(packed: PackedTiles, N: int, np_: int, n_cta: int, mode: int, chunk_tiles: int = 0,
              woff: Optional[torch.Tensor] = None, row_cost: int = ROW_COST) -> Plan:
    """Cut the tile stream of ``packed`` into ``n_cta`` shares, or deal its rows out, on the device (void_plan_segments)."""
    lib = _lib.load()
    dev = packed.row_ptr.device
    panels = (N + PANEL - 1) // PANEL
    n_chunks = (panels + np_ - 1) // np_
    with torch.cuda.device(dev):
        cap = lib.void_plan_capacity(packed.nnz, packed.nbr, n_chunks, n_cta, mode, chunk_tiles)
        segs = torch.empty(cap * 8, dtype=torch.int32, device=dev)
        cta_seg_ptr = torch.empty(n_cta + 1, dtype=torch.int32, device=dev)
        counts = torch.zeros(4, dtype=torch.int32, device=dev)
        ws_bytes = lib.void_plan_ws_bytes(packed.nbr, n_cta)
        ws = torch.empty(ws_bytes, dtype=torch.uint8, device=dev)
        _lib.check(lib.void_plan_segments(_lib.ptr(packed.row_ptr), packed.nbr, n_chunks, n_cta, mode, chunk_tiles,
                                          row_cost, _lib.ptr(woff), _lib.ptr(segs), cap, _lib.ptr(cta_seg_ptr), _lib.ptr(counts),
                                          _lib.ptr(ws), ws_bytes, _lib.stream_ptr(dev)), "void_plan_segments")
        n_segs, n_slots, n_ctr, overflow = (int(x) for x in counts.tolist())
        if overflow:
            raise _lib.VoidB200Error("void_plan_segments: segment list overflow")
        partials = None
        if n_ctr:   # one int32 accumulator per split row; the kernel leaves it zero again
            partials = torch.zeros(n_ctr * np_ * PANEL * TILE, dtype=torch.int32, device=dev)
        counters = torch.zeros(max(n_ctr, 1), dtype=torch.int32, device=dev)
    plan = Plan(segs, cta_seg_ptr, n_cta, np_, n_chunks, n_segs, n_slots, n_ctr, partials, counters, mode,
                chunk_tiles, packed.row_ptr, shape=packed.shape)
    _LIVE_PLANS.add(plan)
    return plan


def prepare_b(b: torch.Tensor, elem_bytes: int = 1) -> torch.Tensor:
    """B as the kernels need it: row-major, rows starting on 16-byte boundaries (the copy engine's rule)."""
    if b.element_size() != elem_bytes:
        raise _lib.VoidB200Error("B must have %d-byte elements to match A, got %s" % (elem_bytes, b.dtype))
    per16 = 16 // elem_bytes
    if b.stride(1) != 1 or b.stride(0) % per16 != 0 or b.data_ptr() % 16 != 0 or b.stride(0) < b.shape[1]:
        K, N = b.shape
        ld = (N + per16 - 1) // per16 * per16
        padded = torch.zeros(K, ld, dtype=b.dtype, device=b.device)
        padded[:, :N] = b
        b = padded[:, :N]
    return b


def spmm(packed: PackedTiles, b: torch.Tensor, out: torch.Tensor, *, scale_mode: int, col_scale=None,
         b_scale: float = 1.0, bias=None, act: int = 0, acc_out=None, plan: Optional[Plan] = None,
         worker_partials=None, use_row_scale: bool = True, panels_per_item: int = 0, stages: int = 0,
         grid: int = 0, tiles_per_stage: int = 0, cta_shape: int = 0, trace=None, flags: int = 0,
         row_bias=None, transposed: bool = False, test_hooks: int = 0, sorted_rows: Optional[bool] = None) -> torch.Tensor:
    """One launch of void_spmm_i8 / void_spmm_f8 / void_spmm_fp on the current stream of b's device.
    With ``transposed`` b is [N, K] and out is [N, M]: the product is out = b @ A^T, both used as they lie.
    The operators call the native host path directly; this form names every option of a launch and takes the
    fields of ``packed`` as they are at the call."""
    opts = (None if plan is None else plan.native_args(), acc_out, worker_partials, panels_per_item, stages, grid,
            tiles_per_stage, cta_shape, trace, flags, test_hooks, sorted_rows, use_row_scale)
    return _lib.native().spmm(packed.new_handle(), b, out, None, scale_mode == _lib.SCALE_PER_TILE, col_scale, b_scale, bias,
                              row_bias, act, transposed, opts)
