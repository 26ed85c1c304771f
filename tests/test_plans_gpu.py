"""Work plans of power-law products: which tile list they were made for, and how long graphs may read them."""
import ctypes

import pytest
import torch

import void_b200 as void
from void_b200 import _lib, _spmm, stream_k, workloads

pytestmark = pytest.mark.gpu


def _case(kind, seed, mean=8.0, n=160):
    w = workloads.block_sparse(workloads.zipf_mask(40, 64, 1.5, 60, mean, seed=seed), n, seed=seed)
    if kind == "fp32":
        return w.a, lambda t, table=None, out=None: void.void_spmm_stream_k(t, w.b, table, out)
    b, scale = void.quantize_cols_int8(w.b)
    return (void.quantize_void_tensor(w.a),
            lambda t, table=None, out=None: void.void_spmm_stream_k(t, b, table, out, b_scale=scale, out_dtype=torch.float16))


def _replace(t, other):
    """The fields of another tensor of the same shape."""
    for name in ("values", "scales", "zero_points", "block_rows", "block_cols", "morton_codes", "n_blocks"):
        if hasattr(t, name):
            setattr(t, name, getattr(other, name))


def _same(kind, x, y):
    if kind == "fp32":                                  # (sums of split rows depend on the order of arrival)
        torch.testing.assert_close(x, y, rtol=1e-5, atol=1e-4)
    else:
        assert torch.equal(x, y)


@pytest.mark.parametrize("kind", ["int8", "fp32"])
@pytest.mark.parametrize("mean", [4.0, 16.0])
@pytest.mark.parametrize("warm,captured", [(False, False), (False, True), (True, False), (True, True)])
def test_a_capture_refuses_the_plan_of_an_earlier_tile_list(kind, mean, warm, captured):
    """The refusal is the host's, before the product would be launched."""
    t, product = _case(kind, 2)
    table = void.compute_stream_k_workload(t)
    product(t, table if warm else None)
    other = _case(kind, 3, mean)[0]
    assert (other.n_blocks > t.n_blocks) == (mean > 8.0)
    _replace(t, other)
    torch.cuda.synchronize()
    with pytest.raises(void.VoidB200Error, match="inside a stream capture"):
        with torch.cuda.graph(torch.cuda.CUDAGraph()):
            product(t, table if captured else None)
    _same(kind, product(t), product(other))
    void.check_device_status()


@pytest.mark.parametrize("kind", ["int8", "fp32"])
def test_a_capture_after_an_edit_of_the_tiles_alone(kind):
    t, product = _case(kind, 4)
    product(t)
    (t.scales if kind == "int8" else t.values).mul_(2)
    want = product(t)
    (t.scales if kind == "int8" else t.values).mul_(2)
    out, graph = torch.empty_like(want), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        product(t, None, out)
    graph.replay()
    torch.cuda.synchronize()
    _same(kind, out, want * 2)
    void.check_device_status()


@pytest.mark.parametrize("how", ["edited tiles", "another operand type"])
def test_a_graph_keeps_its_plan_when_the_tensor_is_packed_again(how):
    t, _ = _case("fp32", 5) if how == "another operand type" else _case("int8", 5)
    n = 160
    b = torch.randint(-3, 4, (t.shape[1], n), device="cuda")
    if how == "another operand type":
        t, b = t.to_dtype(torch.float16), b.half()
        t.values.round_()                               # whole numbers: sums do not depend on the order
        product = lambda out=None: void.void_spmm_stream_k(t, b, out=out)
    else:
        b = b.to(torch.int8)
        product = lambda out=None: void.void_spmm_stream_k(t, b, out=out)
    product()
    if how == "edited tiles":
        t.scales.mul_(2)
    torch.cuda.synchronize()
    plan = next(iter(t._plan_cache.values()))
    out, graph = torch.empty(t.shape[0], n, dtype=b.dtype if b.is_floating_point() else torch.float32, device="cuda"), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        product(out)
    want = product()
    if how == "another operand type":
        void.void_spmm(t, b.float())
    assert not any(p is plan for p in t._plan_cache.values())
    assert any(p is plan for _, plans in t._captured_stores for p in plans)
    del plan
    junk = [torch.full((k,), 0x55, dtype=torch.uint8, device="cuda") for k in (512, 4096, 1 << 14, 1 << 16, 1 << 18) for _ in range(40)]
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want) and len(junk) == 200
    void.check_device_status()


@pytest.mark.parametrize("kind", ["int8", "fp32"])
def test_a_capture_without_a_table_takes_the_plan_that_was_made_along_one(kind):
    """Beyond 1024 CTAs shares are cut along a table either way; one that is given is not kept on the tensor."""
    w = workloads.block_sparse(workloads.zipf_mask(40, 64, 1.5, 60, 8.0, seed=6), 160, seed=6)
    t, b, scale = w.a, w.b, None
    if kind == "int8":
        t = void.quantize_void_tensor(w.a)
        b, scale = void.quantize_cols_int8(w.b)
    want = void.void_spmm_stream_k(t, b, void.compute_stream_k_workload(t), b_scale=scale, n_cta=1025)
    out, graph = torch.empty_like(want), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        void.void_spmm_stream_k(t, b, None, out, b_scale=scale, n_cta=1025)
    graph.replay()
    torch.cuda.synchronize()
    _same(kind, out, want)
    void.check_device_status()


# ------------------------------------------------------------------------------------------ the plan of a product without a table
DROP_FIRST_GROUP = 1 << 16      # test hook: the producers never deliver a CTA's first group of tiles


def _dealt():
    w = workloads.block_sparse(workloads.zipf_mask(64, 256, 1.5, 200, 10.0, seed=7), 256, seed=7)
    q = void.quantize_void_tensor(w.a)
    b, scale = void.quantize_cols_int8(w.b)
    product = lambda: void.void_spmm_stream_k(q, b, b_scale=scale, out_dtype=torch.float16, n_cta=48)
    want = product()
    plan = stream_k.stream_k_plan(q, 256, None, n_cta=48)
    assert plan is next(iter(q._plan_cache.values())) and plan.mode == 3 and plan.n_counters >= 2
    void.check_device_status()
    return q, b.contiguous(), scale, product, want, plan


def test_a_dealt_launch_that_gave_up_leaves_no_partial_sums_behind():
    """The wait for the ring is limited to 5 ms."""
    q, b, scale, product, want, plan = _dealt()
    _spmm.spmm(q.packed(), b, torch.zeros_like(want), scale_mode=_lib.SCALE_ROW_MEAN, col_scale=scale, plan=plan, test_hooks=DROP_FIRST_GROUP | 5)
    torch.cuda.synchronize()
    with pytest.raises(void.VoidB200Error, match="wait gave up"):
        void.check_device_status()
    assert not plan.partials.any() and not plan.counters.any()
    assert torch.equal(product(), want)
    void.check_device_status()


def test_a_dealt_plan_that_points_outside_its_scratch_is_reported_not_followed():
    q, b, scale, product, want, plan = _dealt()
    room = (plan.n_counters - 1) * plan.np * 128 * 32                 # for one split row less than the plan needs
    guard = torch.zeros(room + plan.np * 128 * 32 + 4096, dtype=torch.int32, device="cuda")
    short = _spmm.Plan(plan.segs, plan.cta_seg_ptr, plan.n_cta, plan.np, plan.n_chunks, plan.n_segs, plan.n_slots, plan.n_counters,
                       guard[:room], torch.zeros_like(plan.counters), plan.mode, plan.chunk_tiles)
    _spmm.spmm(q.packed(), b, torch.zeros_like(want), scale_mode=_lib.SCALE_ROW_MEAN, col_scale=scale, plan=short)
    torch.cuda.synchronize()
    assert not guard[room:].any()
    with pytest.raises(void.VoidB200Error, match="does not fit"):
        void.check_device_status()
    assert torch.equal(product(), want)
    void.check_device_status()


def test_a_dealt_plan_with_scratch_inside_the_library():
    q, b, scale, product, want, plan = _dealt()
    for _ in range(2):
        out = torch.full_like(want, float("nan"))
        p, a = q.packed(), _lib.SpmmArgs()
        a.tiles, a.tile_cols, a.tile_scales = p.tiles.data_ptr(), p.tile_cols.data_ptr(), p.tile_scales.data_ptr()
        a.row_ptr, a.row_scale, a.nbr, a.nbc, a.nnz = p.row_ptr.data_ptr(), p.row_scale.data_ptr(), p.nbr, p.nbc, p.nnz
        a.b, a.ldb, a.K, a.N, a.col_scale, a.b_scale = b.data_ptr(), b.stride(0), b.shape[0], b.shape[1], scale.data_ptr(), 1.0
        a.out, a.ldc, a.M, a.out_dtype, a.scale_mode = out.data_ptr(), out.stride(0), out.shape[0], _lib.OUT_DTYPE_CODE[out.dtype], _lib.SCALE_ROW_MEAN
        a.segs, a.cta_seg_ptr, a.n_cta, a.panels_per_item = plan.segs.data_ptr(), plan.cta_seg_ptr.data_ptr(), plan.n_cta, plan.np
        a.status = _lib.status_word(out.device).data_ptr()
        _lib.check(_lib.load().void_spmm_i8_static_scratch(ctypes.byref(a), plan.n_counters, _lib.stream_ptr()), "void_spmm_i8_static_scratch")
        torch.cuda.synchronize()
        void.check_device_status()
        assert torch.equal(out, want)
