"""What a tensor keeps beside its own fields (packed store, tile index, group stores, plans) under a second stream, a second
thread and a stream capture."""
import gc
import threading

import pytest
import torch

import void_b200 as void
from void_b200 import workloads

pytestmark = pytest.mark.gpu

BUSY = 1_000_000_000     # clocks a stream is kept busy: half a second, far longer than the host work behind it takes


def _blocks_handed_out(nbytes, count):
    """Start addresses of ``count`` new blocks of the allocator that hold ``nbytes`` each (kept alive by the tensors)."""
    ts = [torch.zeros(nbytes, dtype=torch.uint8, device="cuda") for _ in range(count)]
    return ts, {t.data_ptr() for t in ts}


# ------------------------------------------------------------------------------------------ lifetime
def test_arrays_of_a_dropped_tensor_wait_for_the_other_stream_that_reads_them():
    w = workloads.block_sparse(workloads.uniform_mask(64, 64, 0.5, seed=1), 256, seed=1)
    q = void.quantize_void_tensor(w.a)
    bq, bs = void.quantize_cols_int8(w.b)
    want = void.void_spmm_int8(q, bq, bs, out_dtype=torch.float16)
    torch.cuda.synchronize()
    p = q.packed()
    arrays = [t.untyped_storage() for t in (p.tiles, p.tile_cols, p.row_ptr, p.row_scale, p.row_order)]
    held = [(s.data_ptr(), s.nbytes()) for s in arrays]
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        out = torch.empty_like(want)
        torch.cuda._sleep(BUSY)
        void.void_spmm_int8(q, bq, bs, out)
    del q, p, arrays
    gc.collect()
    kept = []
    for ptr, nbytes in held:
        ts, starts = _blocks_handed_out(nbytes, 4 if nbytes > 1 << 20 else 64)
        kept += ts
        assert not side.query() and ptr not in starts
    side.synchronize()
    assert torch.equal(out, want)
    void.check_device_status()


def test_index_arrays_of_a_dropped_layer_wait_for_the_other_stream_that_reads_them():
    from void_b200 import autograd
    w = workloads.block_sparse(workloads.uniform_mask(40, 24, 0.5, seed=2), 8, seed=2)
    layer = void.SparseLinear(24 * 32, 40 * 32, w.a, bias=True)
    x = torch.randn(100, 24 * 32, device="cuda")
    with torch.no_grad():
        want = layer(x)
        torch.cuda.synchronize()
        held = autograd._structure(w.a.block_rows, w.a.block_cols, w.a.shape, w.a.n_blocks)[1].untyped_storage()
        ptr, nbytes = held.data_ptr(), held.nbytes()
        side = torch.cuda.Stream()
        with torch.cuda.stream(side):
            torch.cuda._sleep(BUSY)
            got = layer(x)
    autograd._STRUCTURE.clear()
    del held, layer
    gc.collect()
    kept, starts = _blocks_handed_out(nbytes, 64)
    assert not side.query() and ptr not in starts
    side.synchronize()
    assert torch.equal(got, want)
    void.check_device_status()


# ------------------------------------------------------------------------------------------ group stores
GROUPED = [torch.int8, torch.float16, torch.bfloat16, torch.float32]


def _grouped_case(dtype, seed):
    """A tensor and an operand whose products a group store serves, of random values: a changed order of additions shows."""
    w = workloads.block_sparse(workloads.uniform_mask(157, 61, 0.1, seed=seed), 1500, seed=seed)
    if dtype == torch.int8:
        q = void.quantize_void_tensor(w.a)
        bq, bs = void.quantize_cols_int8(w.b)
        return q, lambda out=None: void.void_spmm_int8(q, bq, bs, out, out_dtype=torch.float32), lambda: q.packed()
    from void_b200 import ops
    a, b = w.a.to_dtype(dtype), w.b.to(dtype)
    return a, lambda out=None: void.void_spmm(a, b, out), lambda: ops.packed_fp(a, ops.product_kind(a, b))


def _stores(packed, allowed=None):
    from void_b200 import _lib
    return _lib.native().packed_grouped(packed().native, allowed)


@pytest.mark.parametrize("dtype", GROUPED)
def test_a_group_store_is_built_behind_a_product_and_changes_no_bit(dtype):
    warm, product, _ = _grouped_case(dtype, 2)              # kernels loaded, and memory for a store at hand
    for _ in range(4):
        product()
        torch.cuda.synchronize()
    del warm, product, _
    a, product, packed = _grouped_case(dtype, 3)
    want = product()
    product()
    torch.cuda.synchronize()
    assert _stores(packed) == (True, 0, 0)
    torch.cuda._sleep(BUSY)
    third, fourth = product(), product()
    assert not torch.cuda.current_stream().query()          # the host did not wait for the store
    assert _stores(packed) == (True, 1, 0)                  # and the products did not use it
    torch.cuda.synchronize()
    fifth = product()
    assert _stores(packed) == (True, 1, 1)
    for got in (third, fourth, fifth):
        assert torch.equal(got, want)
    void.check_device_status()


@pytest.mark.parametrize("dtype", GROUPED)
def test_group_stores_can_be_refused_and_are_given_back(dtype):
    a, product, packed = _grouped_case(dtype, 4)
    want = product()
    for _ in range(4):
        product()
    torch.cuda.synchronize()
    product()
    assert _stores(packed) == (True, 1, 1)
    before = torch.cuda.memory_allocated()
    void.allow_group_stores(a, False)
    assert _stores(packed) == (False, 0, 0) and before - torch.cuda.memory_allocated() > a.values.numel() * a.values.element_size()
    for _ in range(4):
        assert torch.equal(product(), want)
    assert _stores(packed) == (False, 0, 0)
    void.allow_group_stores(a, True)
    for _ in range(4):
        product()
    torch.cuda.synchronize()
    assert torch.equal(product(), want) and _stores(packed) == (True, 1, 1)
    c, again, packed_c = _grouped_case(dtype, 4)            # refused before anything is packed
    void.allow_group_stores(c, False)
    for _ in range(4):
        assert torch.equal(again(), want)
    assert _stores(packed_c) == (False, 0, 0)
    void.check_device_status()


@pytest.mark.parametrize("dtype", GROUPED)
def test_group_stores_with_two_streams(dtype):
    a, product, packed = _grouped_case(dtype, 5)
    void.allow_group_stores(a, False)
    want = product()
    void.allow_group_stores(a, True)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    got = []
    for i in range(12):                                     # the build falls between products of both streams
        with torch.cuda.stream(streams[i % 2]):
            if i < 4:
                torch.cuda._sleep(1_000_000)
            got.append(product())
    torch.cuda.synchronize()
    assert all(torch.equal(g, want) for g in got)
    with torch.cuda.stream(streams[1]):                     # dropped while a product on the other stream reads it
        torch.cuda._sleep(BUSY)
        last = product()
    assert _stores(packed) == (True, 1, 1)
    before = torch.cuda.memory_allocated()
    void.allow_group_stores(a, False)
    kept, _ = _blocks_handed_out(before - torch.cuda.memory_allocated(), 2)
    for t in kept:
        t.fill_(0)
    torch.cuda.synchronize()
    assert torch.equal(last, want)
    void.check_device_status()


@pytest.mark.parametrize("dtype", GROUPED)
def test_group_stores_with_two_threads(dtype):
    a, product, packed = _grouped_case(dtype, 6)
    void.allow_group_stores(a, False)
    want = product()
    void.allow_group_stores(a, True)
    torch.cuda.synchronize()
    got, failed = [[], []], []

    def work(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(20):
                    got[k].append(product())
                torch.cuda.current_stream().synchronize()
        except Exception as e:          # noqa: BLE001 - reported below
            failed.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed and all(torch.equal(g, want) for g in got[0] + got[1])
    assert _stores(packed)[1] == 1
    void.check_device_status()


@pytest.mark.parametrize("dtype", GROUPED)
def test_group_stores_and_captures(dtype):
    a, product, packed = _grouped_case(dtype, 7)
    want = product()
    out = [torch.empty_like(want) for _ in range(2)]
    torch.cuda.synchronize()

    def capture(o):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            for _ in range(4):
                product(o)
        return g

    before = capture(out[0])                                # nothing is built while a stream is captured
    assert _stores(packed) == (True, 0, 0)
    for _ in range(4):
        product()
    torch.cuda.synchronize()
    during = capture(out[1])                                # built, but not yet known to be complete: not used
    assert _stores(packed)[1] == 1
    product()
    after_out = torch.empty_like(want)
    after = capture(after_out)
    assert _stores(packed) == (True, 1, 1)
    for g in (before, during, after):
        g.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(o, want) for o in out + [after_out])
    void.check_device_status()


# ------------------------------------------------------------------------------------------ split rows of a work plan
def _split_case(floating=False):
    mask = workloads.zipf_mask(64, 256, 1.5, 200, 10.0, seed=7)
    w = workloads.block_sparse(mask, 256, seed=7)
    if floating:
        return w.a, lambda out=None: void.void_spmm_stream_k(w.a, w.b, out=out, n_cta=48)
    q = void.quantize_void_tensor(w.a)
    bq, bs = void.quantize_cols_int8(w.b)
    return q, lambda out=None: void.void_spmm_stream_k(q, bq, b_scale=bs, out=out, out_dtype=torch.float16, n_cta=48)


@pytest.mark.parametrize("floating", [False, True])
def test_split_rows_on_two_streams_at_once(floating):
    a, product = _split_case(floating)
    want = product()
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    got = []
    for _ in range(2):
        start = torch.cuda.Event()
        torch.cuda._sleep(20_000_000)                       # both streams have their launches queued when they start
        start.record()
        for s in streams:
            s.wait_event(start)
        for _ in range(50):
            for s in streams:
                with torch.cuda.stream(s):
                    got.append(product())
    torch.cuda.synchronize()
    for g in got:
        if floating:                                        # (fp32 sums of split rows depend on the order of arrival)
            torch.testing.assert_close(g, want, rtol=1e-5, atol=1e-5 * float(want.abs().max()))
        else:
            assert torch.equal(g, want)
    (plan,) = a._plan_cache.values()
    assert len(plan.scratch) == 3 and not any(bool(c.any()) or bool(p.any()) for p, c in plan.scratch.values())
    void.check_device_status()


def test_split_rows_in_a_graph_beside_launches_on_other_streams():
    q, product = _split_case()
    want = product()
    torch.cuda.synchronize()
    out = torch.empty_like(want)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        for _ in range(20):
            product(out)
    side = torch.cuda.Stream()
    got = []
    for _ in range(5):
        torch.cuda._sleep(5_000_000)
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            g.replay()
        got += [product() for _ in range(20)]
        side.synchronize()
        assert torch.equal(out, want)
    torch.cuda.synchronize()
    assert all(torch.equal(x, want) for x in got)
    (plan,) = q._plan_cache.values()
    assert len(plan.scratch) == 2 and not any(bool(c.any()) or bool(p.any()) for p, c in plan.scratch.values())
    void.check_device_status()


@pytest.mark.parametrize("dtype", GROUPED)
def test_a_refused_group_store_that_a_graph_reads_stays(dtype):
    a, product, packed = _grouped_case(dtype, 8)
    want = product()
    for _ in range(4):
        product()
    torch.cuda.synchronize()
    product()
    assert _stores(packed) == (True, 1, 1)
    out = torch.empty_like(want)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        product(out)
    before = torch.cuda.memory_allocated()
    void.allow_group_stores(a, False)
    assert _stores(packed) == (False, 0, 0) and torch.cuda.memory_allocated() == before
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want) and torch.equal(product(), want)
    void.check_device_status()
