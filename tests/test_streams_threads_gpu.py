"""What a tensor keeps beside its own fields (packed store, tile index, group stores, plans) under a second stream, a second
thread and a stream capture."""
import gc
import threading

import pytest
import torch

import void_b200 as void
from void_b200 import workloads

pytestmark = pytest.mark.gpu

BUSY = 400_000_000     # clocks a stream is kept busy: 0.2 s, far longer than the host work behind it takes


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
