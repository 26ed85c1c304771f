"""Stream-K load balancing for power-law tile-row lengths on B200.

Mirrors StreamKWorkload (void/stream_k.py:13-33), compute_stream_k_workload (:36-110),
void_spmm_stream_k (:233-301) and analyze_workload_balance (:467-492).

The worker table is the reference's, bit for bit, but it is built by a device kernel instead of a
Python loop with one .item() per row (:76-97).  The SpMM differs in how partial rows are joined:
the reference lets every partial worker lock the output tile and read-modify-write it in the
output dtype (:198-219, an unbounded spin); here rows that are shared between CTAs add their
partial sums into one accumulator per row with atomic adds, and the CTA that arrives last reads it
back and runs the epilogue - no lock and no wait.  Without a table, whole rows and pieces of the
heavy ones are dealt to the CTAs by weight (csrc/plan.cu, mode 3).  With one, the rows in order are
cut into contiguous shares at the table's chunk boundaries (mode 1): consecutive workers of a row
that land on the same CTA keep accumulating in tensor memory.  The result is the same, the dealt
plan is the faster one; products of more segments than one block can sort take shares either way.
For an Int8VOIDTensor the sums are int32, exact and
independent of arrival order; for a floating VOIDTensor (the reference's own argument type) they
are fp32 and their last bits depend on the order, as the reference's locked adds do.
"""
from dataclasses import dataclass
from typing import Optional

import torch

from . import _lib, _spmm
from .format import VOIDTensor
from .int_quant import Int8VOIDTensor, _resolve_b


@dataclass
class StreamKWorkload:
    """Per-worker assignments (void/stream_k.py:13-33)."""
    worker_rows: torch.Tensor          # [n_workers] int32
    worker_block_start: torch.Tensor   # [n_workers] int32
    worker_block_end: torch.Tensor     # [n_workers] int32
    worker_needs_atomic: torch.Tensor  # [n_workers] bool
    n_workers: int
    total_work: int
    # extras used by the B200 launch (not part of the reference dataclass)
    chunk_tiles: int = 0
    worker_offsets: Optional[torch.Tensor] = None


def compute_stream_k_workload(void_tensor, n_workers: Optional[int] = None,
                              max_work_per_worker: int = 16) -> StreamKWorkload:
    """Stream-K work distribution (void/stream_k.py:36-110): rows in order, every non-empty row cut
    into chunks of target = min(ceil(n_blocks / n_workers), max_work_per_worker) tiles."""
    row_ptr, _ = void_tensor.get_row_block_info()
    nbr = void_tensor.block_grid[0]
    rows, start, end, atomic, woff, target = _spmm.streamk_table(row_ptr, nbr, void_tensor.n_blocks, n_workers,
                                                                  max_work_per_worker)
    return StreamKWorkload(worker_rows=rows, worker_block_start=start, worker_block_end=end,
                           worker_needs_atomic=atomic, n_workers=rows.numel(), total_work=void_tensor.n_blocks,
                           chunk_tiles=target, worker_offsets=woff)


def _plan_for(a, packed, N: int, workload: Optional[StreamKWorkload], per_worker: bool, n_cta: Optional[int]):
    """The plan for N columns, kept on the tensor: cut along the worker table where one is given or its workers' sums are asked
    for, else dealt out, which needs no table, as long as that can be (split_mode)."""
    sms = packed.sms
    np_ = _spmm.default_panels(packed.nbr, N, sms) if _lib.KIND_ELEM_BYTES[packed.kind] == 1 else 1
    if n_cta is None:
        n_cta = sms * 4          # four slim CTAs per SM
    n_chunks = (N + _spmm.PANEL * np_ - 1) // (_spmm.PANEL * np_)
    mode = 2 if per_worker else (1 if workload is not None else _spmm.split_mode(packed.nbr, n_chunks, n_cta))
    if mode != 3 and workload is None:
        workload = _cached_workload(a, packed)   # (none inside a capture, unless it is kept)
    chunk_tiles, offsets = (0, None) if mode == 3 or workload is None else (workload.chunk_tiles, workload.worker_offsets)
    key = ("streamk", packed.kind, N, np_, n_cta, mode, chunk_tiles)
    cache = getattr(a, "_plan_cache", None)
    if cache is None:
        cache = a._plan_cache = {}
    plan = cache.get(key)
    if plan is not None and plan.serves(a, packed):
        return plan
    if torch.cuda.is_current_stream_capturing():
        # Nothing can be built here: a plan of either kind that is kept for this width and this tile list does as well.
        if not per_worker:   # (another thread may be adding one for a further width)
            plan = next((p for k, p in list(cache.items()) if k[:5] == key[:5] and k[5] in (1, 3) and p.serves(a, packed)), None)
            if plan is not None:
                return plan
        raise _lib.VoidB200Error("a work plan cannot be built inside a stream capture: multiply the tensor once, with %d columns "
                                 "and its tile list as it is now, before the capture" % N)
    plan = _spmm.make_plan(packed, N, np_, n_cta, mode, chunk_tiles, offsets)
    plan.tile_list = _lib.native().identity(a.block_rows, a.block_cols)
    cache[key] = plan
    return plan


def _require_room(worker_partials, plan, N: int) -> None:
    """Every segment of the plan writes its sums, 32 rows of N."""
    if worker_partials is not None and worker_partials.numel() < plan.n_segs * _spmm.TILE * N:
        raise _lib.VoidB200Error("worker_partials must have %d elements (%d segments), got %d"
                                 % (plan.n_segs * _spmm.TILE * N, plan.n_segs, worker_partials.numel()))


def void_spmm_stream_k(a: Int8VOIDTensor, b: torch.Tensor, workload: Optional[StreamKWorkload] = None,
                       out: Optional[torch.Tensor] = None, *, b_scale=None, out_dtype: Optional[torch.dtype] = None,
                       activation: int = 0, bias: Optional[torch.Tensor] = None,
                       worker_partials: Optional[torch.Tensor] = None, acc_out: Optional[torch.Tensor] = None,
                       n_cta: Optional[int] = None) -> torch.Tensor:
    """Load-balanced SpMM (void/stream_k.py:233-301): a floating VOIDTensor as in the reference, or an
    Int8VOIDTensor with the fused epilogue of void_spmm_int8 (``b_scale`` / ``out_dtype`` apply to it).

    ``worker_partials`` (int32 [n_segments, 32, N], see the plan's segment list) makes every worker of
    the table a segment of its own and records its partial sum - the check that the sum of the
    partials is the row accumulator.

    Inside a stream capture the product takes a work plan that is kept for its width and its tile
    list; where there is none it is refused (so is a list made in inference mode, which leaves no trace of
    its edits).  A replay of a product that was packed inside its capture needs the list as it was then.
    """
    assert b.dim() == 2
    assert a.shape[1] == b.shape[0]
    _lib.require_cuda(a.values, b)
    if isinstance(a, VOIDTensor):
        return _stream_k_fp(a, b, workload, out, activation, bias, worker_partials, acc_out, n_cta)
    if not isinstance(a, Int8VOIDTensor):
        raise TypeError("void_spmm_stream_k takes a VOIDTensor or an Int8VOIDTensor, got %s" % type(a).__name__)
    b_q, scalar, col_scale = _resolve_b(b, b_scale)
    packed = a.packed()
    opts = None
    if a.n_blocks != 0:
        plan = _plan_for(a, packed, b.shape[1], workload, worker_partials is not None, n_cta)
        _require_room(worker_partials, plan, b.shape[1])
        opts = plan.options(acc_out, worker_partials)
    return _lib.native().spmm(packed.native, b_q, out, out_dtype or torch.float32, False, col_scale, scalar, bias, None,
                              activation, False, opts)


def _cached_workload(a, packed) -> Optional[StreamKWorkload]:
    """The table depends on A's structure only: built once per tile index, then reused.  Its size is read back, so that inside a
    stream capture there is only the one that is kept."""
    row_ptr, workload = getattr(a, "_streamk_workload_cache", (None, None))
    if row_ptr is not packed.row_ptr or workload.total_work != a.n_blocks:
        if torch.cuda.is_current_stream_capturing():
            return None
        workload = compute_stream_k_workload(a)
        a._streamk_workload_cache = packed.row_ptr, workload
    return workload


def _stream_k_fp(a: VOIDTensor, b, workload, out, activation, bias, worker_partials, acc_out, n_cta):
    """void_spmm_stream_k on a floating VOIDTensor (void/stream_k.py:233-301): result in B's dtype."""
    from . import ops
    if a.n_blocks == 0:
        return ops.void_spmm(a, b, out, activation=activation, bias=bias)
    packed = ops.packed_fp(a, ops.product_kind(a, b))
    plan = _plan_for(a, packed, b.shape[1], workload, worker_partials is not None, n_cta)
    _require_room(worker_partials, plan, b.shape[1])
    return ops.void_spmm(a, b, out, activation=activation, bias=bias, plan=plan, acc_out=acc_out,
                         worker_partials=worker_partials)


def stream_k_plan(a, N: int, workload: Optional[StreamKWorkload], per_worker: bool = False, n_cta: Optional[int] = None,
                  kind: Optional[int] = None) -> _spmm.Plan:
    """The device-built work plan that void_spmm_stream_k uses for an N-column product with this ``workload``; None: without
    one, which is another plan (``kind``: the product kind of a floating VOIDTensor, fp32 operands by default)."""
    if isinstance(a, VOIDTensor):
        from . import ops
        packed = ops.packed_fp(a, _lib.FP_KIND.get(a.values.dtype, _lib.KIND_TF32) if kind is None else kind)
    else:
        packed = a.packed()
    return _plan_for(a, packed, N, workload, per_worker, n_cta)


def analyze_workload_balance(void_tensor) -> dict:
    """Row-length statistics (void/stream_k.py:467-492)."""
    row_ptr, _ = void_tensor.get_row_block_info()
    row_work = (row_ptr[1:] - row_ptr[:-1]).float()
    non_empty = row_work > 0
    nz = row_work[non_empty]
    if len(nz) == 0:
        return {"empty": True}
    return {
        "empty": False,
        "n_rows": len(row_work),
        "n_nonempty_rows": non_empty.sum().item(),
        "min_blocks_per_row": nz.min().item(),
        "max_blocks_per_row": nz.max().item(),
        "mean_blocks_per_row": nz.mean().item(),
        "std_blocks_per_row": nz.std().item(),
        "imbalance_ratio": (nz.max() / nz.mean()).item(),
        "coefficient_of_variation": (nz.std() / nz.mean()).item(),
    }


__all__ = ["StreamKWorkload", "compute_stream_k_workload", "void_spmm_stream_k", "analyze_workload_balance",
           "stream_k_plan"]
