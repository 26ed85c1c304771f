"""Paths that only run when something is wrong, exercised without any fault, trap or unbounded wait: a bounded
device-side wait that is made to run out (a test hook keeps one ring stage from ever being filled, the wait
limit is set to a few milliseconds), and a work plan that points outside the scratch it was given.  In both the
kernel returns in an orderly way with a code in the status word, and the next launch is correct."""
import pytest
import torch

import void_b200 as void
from void_b200 import _lib, _spmm, stream_k, workloads

pytestmark = pytest.mark.gpu

DROP_FIRST_GROUP = 1 << 16


def _small():
    mask = workloads.zipf_mask(64, 256, 1.5, 200, 10.0, seed=7)
    w = workloads.block_sparse(mask, 256, seed=7)
    q = void.quantize_void_tensor(w.a)
    bq, bs = void.quantize_cols_int8(w.b)
    return q, bq.contiguous(), bs


def test_bounded_wait_runs_out_with_a_status_and_the_next_launch_is_clean():
    q, bq, bs = _small()
    want = void.void_spmm_int8(q, bq, bs, out_dtype=torch.float16)
    torch.cuda.synchronize()
    void.check_device_status()
    out = torch.zeros_like(want)
    # every CTA's first group of tiles is never delivered; the consumer's wait is limited to 5 ms
    _spmm.spmm(q.packed(), bq, out, scale_mode=_lib.SCALE_ROW_MEAN, col_scale=bs, test_hooks=DROP_FIRST_GROUP | 5)
    with pytest.raises(void.VoidB200Error, match="wait gave up"):
        void.check_device_status()
    void.check_device_status()                                   # the word was cleared
    again = void.void_spmm_int8(q, bq, bs, out_dtype=torch.float16)   # tensor memory was given back, nothing hangs
    void.check_device_status()
    assert torch.equal(again, want)


def test_a_launch_that_gave_up_leaves_no_partial_sums_behind():
    q, bq, bs = _small()
    wl = void.compute_stream_k_workload(q)
    want = void.void_spmm_stream_k(q, bq, wl, b_scale=bs, out_dtype=torch.float16, n_cta=48)
    plan = stream_k.stream_k_plan(q, 256, wl, n_cta=48)
    assert plan.n_counters > 0
    void.check_device_status()
    out = torch.zeros_like(want)
    _spmm.spmm(q.packed(), bq, out, scale_mode=_lib.SCALE_ROW_MEAN, col_scale=bs, plan=plan, test_hooks=DROP_FIRST_GROUP | 5)
    torch.cuda.synchronize()
    dirty = bool(plan.partials.any()) or bool(plan.counters.any())
    with pytest.raises(void.VoidB200Error):
        void.check_device_status()
    assert not plan.partials.any() and not plan.counters.any()   # cleared together with the status word
    again = void.void_spmm_stream_k(q, bq, wl, b_scale=bs, out_dtype=torch.float16, n_cta=48)
    void.check_device_status()
    assert torch.equal(again, want), "dirty scratch before the reset: %s" % dirty


def test_plan_that_points_outside_its_scratch_is_reported_not_followed():
    q, bq, bs = _small()
    wl = void.compute_stream_k_workload(q)
    plan = stream_k.stream_k_plan(q, 256, wl, n_cta=48)
    assert plan.n_counters >= 2
    want = void.void_spmm_stream_k(q, bq, wl, b_scale=bs, out_dtype=torch.float16, n_cta=48)
    per_row = plan.np * 128 * 32
    guard = torch.zeros(plan.n_counters * per_row + 4096, dtype=torch.int32, device="cuda")
    short = _spmm.Plan(plan.segs, plan.cta_seg_ptr, plan.n_cta, plan.np, plan.n_chunks, plan.n_segs, plan.n_slots,
                       plan.n_counters, guard[:(plan.n_counters - 1) * per_row], torch.zeros_like(plan.counters),
                       plan.mode, plan.chunk_tiles)                # room for one split row less than the plan needs
    out = torch.zeros_like(want)
    _spmm.spmm(q.packed(), bq, out, scale_mode=_lib.SCALE_ROW_MEAN, col_scale=bs, plan=short)
    torch.cuda.synchronize()
    assert not guard[(plan.n_counters - 1) * per_row:].any()      # nothing was written behind the scratch
    with pytest.raises(void.VoidB200Error, match="does not fit"):
        void.check_device_status()


def _earlier_failure():
    """A call that fails on the host: more shared memory than a block can have.  The runtime remembers its error."""
    assert _lib.load().void_launch_floor(1, 128, 10_000_000, torch.cuda.current_stream().cuda_stream) != 0


@pytest.mark.parametrize("what", ["product", "store", "fp8_exact", "few_columns", "grouped", "stream_k", "columns", "tiles", "index", "long_index", "convert", "linear"])
def test_a_launch_reports_its_own_status_and_no_earlier_calls(what):
    q, bq, bs = _small()
    gen = torch.Generator().manual_seed(5)
    a = void.dense_to_void(torch.randn(512, 512, generator=gen).cuda())
    lib, stream = _lib.load(), torch.cuda.current_stream().cuda_stream
    if what == "linear":
        layer, x = void.SparseLinear(512, 512, a, bias=True), torch.randn(64, 512, generator=gen).cuda().requires_grad_(True)
        call = lambda: layer(x).sum().backward()
    elif what == "grouped":
        big = workloads.block_sparse(workloads.uniform_mask(128, 128, 0.5, seed=1), 2048, seed=1)
        t, b = big.a.to_dtype(torch.float16), big.b.half()
        for _ in range(5):      # the fifth runs the grouped kernel, whose first launch sets its attributes
            torch.cuda.synchronize()
            void.void_spmm(t, b)
        call = lambda: void.void_spmm(t, b)
    else:
        rows, cols = a.block_rows, a.block_cols
        f8 = void.void_tensor_to_fp8(a)
        b8, b8s, _ = void.quantize_cols_fp8(torch.randn(512, 256, generator=gen).cuda())
        b8q, b8qs = void.quantize_cols_int8(torch.randn(512, 256, generator=gen).cuda())
        wide = torch.randperm(700 * 700, generator=gen)[:20000]
        wide_rows, wide_cols = (wide // 700).int().cuda(), (wide % 700).int().cuda()
        from void_b200.format import build_tile_index
        call = {"product": lambda: void.void_spmm_int8(q, bq, bs), "store": lambda: void.void_spmm_int8(void.quantize_void_tensor(a), b8q, b8qs),
                "fp8_exact": lambda: void.void_spmm_fp8(f8, b8, b_scale=b8s, scale_terms=0),
                "few_columns": lambda: void.void_spmv(a, torch.ones(512, device="cuda")),
                "stream_k": lambda: void.void_spmm_stream_k(q, bq, b_scale=bs),
                "columns": lambda: void.quantize_cols_int8(torch.randn(20000, 40, generator=gen).cuda()),
                "tiles": lambda: void.void_tensor_to_fp8(a),
                "index": lambda: build_tile_index(rows, cols, 16, 16),
                "long_index": lambda: build_tile_index(wide_rows, wide_cols, 700, 700),
                "convert": lambda: void.quantize_void_tensor(void.dense_to_void(torch.ones(96, 96, device="cuda"))).packed()}[what]
    call()
    for _ in range(2):          # what the first call builds, and what every one launches
        _earlier_failure()
        call()
    torch.cuda.synchronize()
    void.check_device_status()
