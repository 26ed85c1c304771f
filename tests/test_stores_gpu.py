"""Stores derived from a tensor (packed tiles, tile index, dequantised tiles, plans) follow every change of its fields."""
import pytest
import torch

import void_b200 as void
from void_b200 import workloads

pytestmark = pytest.mark.gpu


def _case(seed, nbr=9, nbc=7, n=40):
    return workloads.block_sparse(workloads.uniform_mask(nbr, nbc, 0.5, seed=seed), n, seed=seed)


def test_tiles_read_in_another_layout_are_packed_again():
    w = _case(1)
    for a in (w.a, w.a.half()):
        b = w.b.to(a.values.dtype)
        void.void_spmm(a, b)
        flipped = void.VOIDTensor(a.values.transpose(1, 2).contiguous(), a.block_rows, a.block_cols, a.morton_codes, a.shape,
                                  (32, 32), 0, a.n_blocks, 0.0)
        want = void.void_spmm(flipped, b)
        a.values = a.values.transpose(1, 2)            # same address, same version
        assert torch.equal(void.void_spmm(a, b), want)


@pytest.mark.parametrize("terms", [0, 2, 3, None])
def test_fp8_scales_that_land_at_the_old_address_are_seen(terms):
    w = _case(2)
    a = void.void_tensor_to_fp8(w.a)
    bq, bs, _ = void.quantize_cols_fp8(w.b)
    if terms is None:                                  # floating B: the dequantised copy
        product = lambda: void.void_spmm_fp8(a, w.b, torch.float32)
    else:
        product = lambda: void.void_spmm_fp8(a, bq, torch.float32, b_scale=bs, scale_terms=terms)
    want = product() * 2
    for _ in range(8):
        new = (a.scaling_info.scale * 2).cpu()
        a.scaling_info.scale = None                    # the block is free before the new tensor is made
        a.scaling_info.scale = new.cuda()
        assert torch.equal(product(), want)
        want = want * 2


def test_tensors_without_versions_are_packed_for_every_product():
    w = _case(3)
    with torch.inference_mode():
        a = void.VOIDTensor(w.a.values.clone(), w.a.block_rows.clone(), w.a.block_cols.clone(), w.a.morton_codes, w.a.shape, (32, 32),
                            0, w.a.n_blocks, 0.0)
        q = void.quantize_void_tensor(a)
        bq, bs = void.quantize_cols_int8(w.b)
        for make in (lambda: void.void_spmm(a, w.b), lambda: void.void_spmm_int8(q, bq, bs)):
            want = make() * 2
            a.values.mul_(2)
            q.scales.mul_(2)
            assert torch.equal(make(), want)


def _swap_rows(t):
    """Tile list of the matrix with its tile rows reversed, edited in place."""
    nbr = t.block_grid[0]
    t.block_rows.mul_(-1).add_(nbr - 1)


@pytest.mark.parametrize("kind", ["fp32", "fp16", "int8", "streamk", "streamk_int8", "linear"])
def test_an_edited_tile_list_is_indexed_again(kind):
    w = _case(4, nbr=12, nbc=20, n=130)
    a, b = w.a, w.b
    if kind == "fp16":
        a, b = a.half(), b.half()
    if kind.endswith("int8"):
        a = void.quantize_void_tensor(a)
        bq, bs = void.quantize_cols_int8(b)
    product = {"fp32": lambda t: void.void_spmm(t, b), "fp16": lambda t: void.void_spmm(t, b),
               "int8": lambda t: void.void_spmm_int8(t, bq, bs), "streamk": lambda t: void.void_spmm_stream_k(t, b, n_cta=16),
               "streamk_int8": lambda t: void.void_spmm_stream_k(t, bq, b_scale=bs, n_cta=16),
               "linear": lambda t: void.void_linear(t, b.t().contiguous()).t()}[kind]
    product(a)
    a.get_row_block_info()
    _swap_rows(a)
    got = product(a)
    fresh = a.to(a.values.device)                      # the same fields, nothing kept
    fresh.block_rows, fresh.block_cols = a.block_rows.clone(), a.block_cols.clone()
    if kind == "streamk":                              # (sums of split rows depend on the order of arrival)
        torch.testing.assert_close(got, product(fresh), rtol=1e-5, atol=1e-4)
    else:
        assert torch.equal(got, product(fresh))
    assert torch.equal(a.get_row_block_info()[0], fresh.get_row_block_info()[0])
    a.block_rows[0] = 100                              # no longer a valid list: refused as it was before anything was kept
    with pytest.raises(ValueError, match="invalid VOID tile list"):
        product(a)
    void.check_device_status()


def test_a_layer_whose_tile_list_is_another_view_of_the_same_memory():
    w = _case(5, nbr=6, nbc=6, n=8)
    n = w.a.n_blocks
    cols = torch.arange(n, dtype=torch.int32, device="cuda") % 6
    rows = torch.arange(n, dtype=torch.int32, device="cuda") // 6
    both = torch.stack([rows, (n - 1) // 6 - rows], 1).reshape(-1).contiguous()                  # rows and reversed rows in turn
    x = torch.randn(5, 192, device="cuda")

    def dense(r):
        out = torch.zeros(6, 6, 32, 32, device="cuda")
        out[r.long(), cols.long()] = w.a.values
        return out.permute(0, 2, 1, 3).reshape(192, 192)

    for r in (both[0::2], both[1::2]):
        y = void.VOIDLinearFunction.apply(w.a.values, r, cols, (192, 192), (32, 32), n, x, None)
        torch.testing.assert_close(y, x @ dense(r).t(), rtol=2e-3, atol=2e-3 * float(y.abs().max()))


@pytest.mark.parametrize("kind", ["fp32", "int8", "fp8", "fp8_exact", "fp8_floating", "linear", "mlp"])
def test_a_tensor_first_used_inside_a_capture(kind):
    w = _case(6)
    a, b = w.a, w.b
    q = {"int8": lambda: void.quantize_void_tensor(a), "fp8": lambda: void.void_tensor_to_fp8(a),
         "fp8_exact": lambda: void.void_tensor_to_fp8(a), "fp8_floating": lambda: void.void_tensor_to_fp8(a)}.get(kind, lambda: a.to(a.values.device))
    bq, bs = void.quantize_cols_int8(b) if kind == "int8" else void.quantize_cols_fp8(b)[:2]
    back = void.VOIDTensor(a.values, a.block_cols, a.block_rows, a.morton_codes, a.shape[::-1], (32, 32), 0, a.n_blocks, 0.0)
    product = {"fp32": lambda t: void.void_spmm(t, b), "int8": lambda t: void.void_spmm_int8(t, bq, bs),
               "fp8": lambda t: void.void_spmm_fp8(t, bq, b_scale=bs),
               "fp8_exact": lambda t: void.void_spmm_fp8(t, bq, b_scale=bs, scale_terms=0),
               "fp8_floating": lambda t: void.void_spmm_fp8(t, b),
               "linear": lambda t: void.void_linear(t, b.t().contiguous()),
               "mlp": lambda t: void.fused_sparse_mlp(b.t().contiguous(), t, back)}[kind]
    want = product(q())
    t = q()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        first, second = product(t), product(t)
    assert torch.equal(product(t), want)               # before the graph has run, its arrays hold nothing
    for _ in range(2):
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(first, want) and torch.equal(second, want)
    assert torch.equal(product(t), want)
    void.check_device_status()


@pytest.mark.parametrize("n", [8, 40, 300])
@pytest.mark.parametrize("kind", ["int8", "fp8_exact"])
def test_first_replays_of_products_packed_inside_a_capture(kind, n):
    """Only the first replay finds arrays that nothing has written: new graphs, their first replay right behind a product."""
    w = _case(8, n=n)
    make, quantise = (void.quantize_void_tensor, void.quantize_cols_int8) if kind == "int8" else (void.void_tensor_to_fp8, void.quantize_cols_fp8)
    bq, bs = quantise(w.b)[:2]
    product = (lambda t: void.void_spmm_int8(t, bq, bs)) if kind == "int8" else (lambda t: void.void_spmm_fp8(t, bq, b_scale=bs, scale_terms=0))
    want, keep = product(make(w.a)), []
    for _ in range(12):
        t, g = make(w.a), torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(g):
            out = product(t)
        product(make(w.a))
        g.replay()
        keep.append((g, t, out))
    assert all(torch.equal(out, want) for _, _, out in keep)
    void.check_device_status()


@pytest.mark.parametrize("how", ["deepcopy", "copy", "file"])
@pytest.mark.parametrize("kind", ["fp32", "int8", "fp8", "fp8_floating", "streamk", "module", "layer"])
def test_tensors_that_were_multiplied_can_be_copied_and_saved(kind, how, tmp_path):
    import copy
    w = _case(7, n=130)
    b, bt = w.b, w.b.t().contiguous()
    bq, bs = void.quantize_cols_fp8(b)[:2] if kind == "fp8" else void.quantize_cols_int8(b)
    t = {"int8": lambda: void.quantize_void_tensor(w.a), "streamk": lambda: void.quantize_void_tensor(w.a),
         "fp8": lambda: void.void_tensor_to_fp8(w.a), "fp8_floating": lambda: void.void_tensor_to_fp8(w.a),
         "module": lambda: void.FusedSparseLinear(224, 288, w.a), "layer": lambda: void.SparseLinear(224, 288, w.a)}.get(kind, lambda: w.a)()
    product = {"fp32": lambda x: void.void_spmm(x, b), "int8": lambda x: void.void_spmm_int8(x, bq, bs),
               "streamk": lambda x: void.void_spmm_stream_k(x, bq, b_scale=bs, n_cta=16),
               "fp8": lambda x: void.void_spmm_fp8(x, bq, b_scale=bs), "fp8_floating": lambda x: void.void_spmm_fp8(x, b),
               "module": lambda x: x(bt), "layer": lambda x: x(bt).detach()}[kind]
    want = product(t)
    if how == "file":
        torch.save(t, tmp_path / "t.pt")
        again = torch.load(tmp_path / "t.pt", weights_only=False)
    else:
        again = getattr(copy, how)(t)
    assert torch.equal(product(again), want) and torch.equal(product(t), want)
    if hasattr(again, "get_row_block_info"):
        assert torch.equal(again.get_row_block_info()[0], t.get_row_block_info()[0])


def test_states_of_earlier_versions_are_read_without_what_they_derived():
    w = _case(8)
    q = void.quantize_void_tensor(w.a)
    bq, bs = void.quantize_cols_int8(w.b)
    want = void.void_spmm_int8(q, bq, bs)
    old = dict(q.__getstate__(), _packed_cache=object(), _plan_cache={1: 2}, _streamk_workload_cache=object())
    again = void.Int8VOIDTensor.__new__(void.Int8VOIDTensor)
    again.__setstate__(old)
    assert torch.equal(void.void_spmm_int8(again, bq, bs), want)


@pytest.mark.parametrize("kind", ["fp32", "int8", "fp8", "fp8_exact", "fp8_floating", "streamk", "spmv", "mlp"])
def test_a_graph_keeps_reading_what_it_was_captured_with(kind):
    w = _case(9, nbr=12, nbc=20, n=130)
    a, b = w.a, w.b
    bq, bs = void.quantize_cols_fp8(b)[:2] if kind.startswith("fp8") else void.quantize_cols_int8(b)
    t = void.void_tensor_to_fp8(a) if kind.startswith("fp8") else (void.quantize_void_tensor(a) if kind in ("int8", "streamk") else a)
    back = void.VOIDTensor(a.values.clone(), a.block_cols, a.block_rows, a.morton_codes, a.shape[::-1], (32, 32), 0, a.n_blocks, 0.0)
    bt = b.t().contiguous()
    product = {"fp32": lambda: void.void_spmm(t, b), "int8": lambda: void.void_spmm_int8(t, bq, bs),
               "fp8": lambda: void.void_spmm_fp8(t, bq, b_scale=bs), "fp8_exact": lambda: void.void_spmm_fp8(t, bq, b_scale=bs, scale_terms=0),
               "fp8_floating": lambda: void.void_spmm_fp8(t, b), "streamk": lambda: void.void_spmm_stream_k(t, bq, b_scale=bs, n_cta=16),
               "spmv": lambda: void.void_spmv(t, b[:, 0].contiguous()), "mlp": lambda: void.fused_sparse_mlp(bt, t, back)}[kind]
    want = product()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = product()
    scale = t.scaling_info.scale if kind.startswith("fp8") else (t.scales if kind in ("int8", "streamk") else t.values)
    for _ in range(2):
        scale.mul_(2)                                  # the tensor's own products follow it ...
        new = product()
    assert not torch.equal(new, want)
    junk = [torch.full((n,), 0x55, dtype=torch.uint8, device="cuda") for n in (512, 4096, 1 << 16, 1 << 18, 1 << 19, 1 << 20) for _ in range(40)]
    g.replay()                                         # ... the graph multiplies what it was captured with
    torch.cuda.synchronize()
    assert torch.equal(out, want) and len(junk) == 240
    assert len(t._captured_stores) == 1
    void.check_device_status()


def test_structures_that_a_graph_reads_are_not_dropped(monkeypatch):
    from void_b200 import autograd
    monkeypatch.setattr(autograd, "_STRUCTURE", {})
    monkeypatch.setattr(autograd, "_STRUCTURE_MAX", 2)
    layers = []
    for seed in range(4):
        w = _case(10 + seed)
        layers.append(void.SparseLinear(224, 288, w.a))
    x = torch.randn(40, 224, device="cuda")
    with torch.no_grad():
        want = layers[0](x)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            out = layers[0](x)
        first = next(iter(autograd._STRUCTURE))
        for layer in layers[1:]:
            layer(x)
        assert len(autograd._STRUCTURE) == 2 and first in autograd._STRUCTURE
        g.replay()
        assert torch.equal(out, want)
    void.check_device_status()
