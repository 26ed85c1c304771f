"""Every kernel variant that a size rule selects, at the sizes where it can go wrong: edges of its tiles, remainders, the
smallest and largest of its range and the first size of the next variant."""
import numpy as np
import pytest
import torch

import void_b200 as void
from oracle import void_oracle as vo

pytestmark = pytest.mark.gpu


# ------------------------------------------------------------------------------------------ columns quantised
@pytest.mark.parametrize("k,n", [(1, 1), (7, 5), (8, 16), (33, 17), (513, 36), (8192, 12), (8193, 288), (8200, 292),
                                 (26624, 40), (26632, 40), (30000, 3)])
def test_quantised_columns_match_the_oracle_bits(k, n):
    gen = torch.Generator().manual_seed(k * 1000 + n)
    b = torch.randn(k, n, generator=gen)
    b[:, 0] = torch.randint(-256, 257, (k,), generator=gen) * 0.5         # scale 1: quotients on half integers ...
    b[0, 0] = 128.0
    if k > 8:
        b[5, 0] = float(np.nextafter(np.float32(2.5), np.float32(3)))
        b[6, 0] = float(np.nextafter(np.float32(-3.5), np.float32(0)))
    b[:, n // 2] *= 0 if n > 1 else 1                                     # ... and a column of zeros
    q, s = void.quantize_cols_int8(b.cuda())
    ref_q, ref_s = vo.quantize_int8_cols(b.numpy())
    assert np.array_equal(s.cpu().numpy(), ref_s) and np.array_equal(q.cpu().numpy(), ref_q)
    f, fs, fi = void.quantize_cols_fp8(b.cuda())
    ref_f, ref_fs, ref_fi = vo.quantize_fp8_cols(b.numpy())
    assert np.array_equal(fs.cpu().numpy(), ref_fs) and np.array_equal(fi.cpu().numpy(), ref_fi)
    assert np.array_equal(f.view(torch.uint8).cpu().numpy(), ref_f)
    off = torch.zeros(k, n + 3).cuda()[:, 1:n + 1]                        # rows that start off 16-byte boundaries
    off.copy_(b)
    assert torch.equal(void.quantize_cols_int8(off)[0], q)


# ------------------------------------------------------------------------------------------ training
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m,k,n", [(32, 32, 1), (64, 96, 31), (96, 160, 64), (200, 168, 65), (320, 264, 130), (40, 72, 515)])
def test_linear_gradients_exact_on_small_integers(dtype, m, k, n):
    gen = torch.Generator().manual_seed(m + k + n)
    nbr, nbc = (m + 31) // 32, (k + 31) // 32
    mask = torch.rand(nbr, nbc, generator=gen) < 0.6
    mask[0, 0] = True
    dense = torch.randint(-2, 3, (m, k), generator=gen).float() * mask.repeat_interleave(32, 0).repeat_interleave(32, 1)[:m, :k]
    a = void.dense_to_void(dense.cuda()).to_dtype(dtype)
    lin = void.SparseLinear(k, m, a, bias=True)
    x = torch.randint(-2, 3, (n, k), generator=gen).cuda().to(dtype).requires_grad_(True)
    gy = torch.randint(-1, 2, (n, m), generator=gen).cuda().to(dtype)
    y = lin(x)
    y.backward(gy)
    void.check_device_status()
    ref = a.to_dense().float().requires_grad_(True)
    xr = x.detach().float().requires_grad_(True)
    yr = xr @ ref.t()
    yr.backward(gy.float())
    assert torch.equal(y.float(), yr.to(dtype).float()) and torch.equal(x.grad.float(), xr.grad.to(dtype).float())
    assert torch.equal(lin.bias.grad.float(), gy.float().sum(0).to(dtype).float())
    grid = torch.zeros(nbr * 32, nbc * 32, device="cuda")
    grid[:m, :k] = ref.grad
    tiles = grid.reshape(nbr, 32, nbc, 32).permute(0, 2, 1, 3)[a.block_rows.long(), a.block_cols.long()]
    assert torch.equal(lin.sparse_weight.values.grad.float(), tiles.to(dtype).float())


# ------------------------------------------------------------------------------------------ format and set-up
@pytest.mark.parametrize("m,n,off,dtype,threshold", [
    (1, 1, 0, torch.float32, 0.0), (31, 33, 0, torch.float32, 0.0), (64, 126, 1, torch.float32, 0.0),
    (100, 130, 0, torch.float16, 2.0), (65, 257, 0, torch.bfloat16, 0.0), (33, 264, 1, torch.bfloat16, 1.5),
    (64, 256, 0, torch.float32, -1.0), (32, 32800, 0, torch.float16, 0.0), (70, 16384, 0, torch.float32, 0.0),
    (70, 16385, 0, torch.bfloat16, 0.0)])
def test_dense_to_void_widths_and_alignments(m, n, off, dtype, threshold):
    gen = torch.Generator().manual_seed(m * 7 + n)
    full = (torch.randn(m, n, generator=gen) * (torch.rand(m, n, generator=gen) < 0.01)).to(dtype)
    wide = torch.zeros(m, n + off, dtype=dtype, device="cuda")
    wide[:, off:] = full.cuda()
    v = void.dense_to_void(wide[:, off:], threshold=threshold)
    f = vo.dense_to_void_fields(full.float().numpy(), threshold=threshold)
    assert v.n_blocks == f["n_blocks"] and v.nnz_original == f["nnz_original"]
    for name in ("block_rows", "block_cols", "morton_codes"):
        assert np.array_equal(getattr(v, name).cpu().numpy(), f[name])
    assert np.array_equal(v.values.float().cpu().numpy(), f["values"])


@pytest.mark.parametrize("nbr,nbc", [(1, 1), (1, 70), (256, 40), (257, 40), (1023, 33), (1025, 2), (4096, 3), (4097, 3), (600, 2100)])
def test_packed_store_of_grids_of_every_size(nbr, nbc):
    gen = torch.Generator().manual_seed(nbr + nbc)
    mask = (torch.rand(nbr, nbc, generator=gen) < min(0.4, 3000 / (nbr * nbc))).numpy()
    mask[0, nbc - 1] = True
    rows, cols = np.nonzero(mask)
    perm = np.random.default_rng(0).permutation(len(rows))
    rows, cols = rows[perm].astype(np.int32), cols[perm].astype(np.int32)
    a = void.VOIDTensor(torch.randn(len(rows), 32, 32).cuda().half(), torch.from_numpy(rows).cuda(), torch.from_numpy(cols).cuda(),
                        torch.zeros(len(rows), dtype=torch.int64, device="cuda"), (nbr * 32, nbc * 32), (32, 32), 0, len(rows), 0.0)
    q = void.quantize_void_tensor(a)                                     # 16-bit tiles are quantised as they are
    ref_q, ref_s = vo.quantize_int8_tiles(a.values.float().cpu().numpy())
    assert np.array_equal(q.values.cpu().numpy(), ref_q) and np.array_equal(q.scales.cpu().numpy(), ref_s)
    assert torch.equal(q.block_rows, a.block_rows) and q.block_rows.data_ptr() != a.block_rows.data_ptr()
    p = q.packed()
    ref_rp, ref_bi = vo.row_block_info(rows, cols, nbr, nbc)
    assert np.array_equal(p.row_ptr.cpu().numpy(), ref_rp) and np.array_equal(p.block_indices.cpu().numpy(), ref_bi)
    assert np.array_equal(p.tile_cols.cpu().numpy(), cols[ref_bi]) and np.array_equal(p.tile_scales.cpu().numpy(), ref_s[ref_bi])
    order = np.argsort(-np.diff(ref_rp), kind="stable")
    assert np.array_equal(p.row_order.cpu().numpy(), order)


@pytest.mark.parametrize("nbr,nbc,nnz", [(1, 1, 1), (1, 1, 0), (3, 33, 60), (4000, 64, 16384), (4001, 64, 900), (363, 1024, 16384),
                                         (363, 1024, 16385), (364, 1024, 1000), (1024, 256, 16000)])
def test_tile_index_around_the_limits_of_one_block(nbr, nbc, nnz):
    from void_b200.format import build_tile_index
    gen = torch.Generator().manual_seed(nbr + nbc + nnz)
    cells = torch.randperm(nbr * nbc, generator=gen)[:nnz]
    rows, cols = (cells // nbc).int(), (cells % nbc).int()
    row_ptr, indices = build_tile_index(rows.cuda(), cols.cuda(), nbr, nbc)
    assert torch.equal(row_ptr.cpu(), torch.cat([torch.zeros(1), torch.bincount(rows.long(), minlength=nbr).cumsum(0)]).int())
    assert torch.equal(indices.cpu(), cells.argsort().int())


def _index_list(nbr, nbc, nnz):
    gen = torch.Generator().manual_seed(nbr + 3 * nbc + nnz)
    cells = torch.randperm(nbr * nbc, generator=gen)[:nnz]
    return cells, (cells // nbc).int().cuda(), (cells % nbc).int().cuda()


@pytest.mark.parametrize("nbr,nbc,nnz", [(128, 128, 8192), (128, 128, 16384), (65, 512, 8192), (65, 512, 8193), (64, 512, 16384), (64, 513, 16385),
                                         (16384, 32, 8192), (16385, 32, 8192), (5461, 96, 8192), (5462, 65, 100), (15, 32768, 8192)])
def test_tile_index_where_one_block_hands_over(nbr, nbc, nnz):
    from void_b200.format import build_tile_index
    cells, rows, cols = _index_list(nbr, nbc, nnz)
    row_ptr, indices = build_tile_index(rows, cols, nbr, nbc)
    assert torch.equal(row_ptr.cpu(), torch.cat([torch.zeros(1), torch.bincount(cells // nbc, minlength=nbr).cumsum(0)]).int())
    assert torch.equal(indices.cpu(), cells.argsort().int())


def test_the_time_of_a_tile_index_does_not_follow_the_width_of_the_grid():
    """The same number of tiles in a square grid and in wide ones of many bitmap words: 1.6 times as long measured, 7 and 20 times
    when every tile added up the words of its row."""
    from void_b200 import _lib
    lib, took = _lib.load(), []
    for nbr, nbc in ((128, 128), (363, 1024), (15, 32768)):
        _, rows, cols = _index_list(nbr, nbc, 8000)
        row_ptr, indices = (torch.empty(n, dtype=torch.int32, device="cuda") for n in (nbr + 1, 8000))
        ws = torch.empty(lib.void_tile_index_ws_bytes(nbr, nbc), dtype=torch.uint8, device="cuda")
        stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            for _ in range(20):
                assert lib.void_build_tile_index(_lib.ptr(rows), _lib.ptr(cols), 8000, nbr, nbc, _lib.ptr(row_ptr), _lib.ptr(indices),
                                                 _lib.ptr(ws), ws.numel(), stream.cuda_stream) == 0
        times = []
        for _ in range(10):
            begin, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            begin.record()
            graph.replay()
            end.record()
            end.synchronize()
            times.append(begin.elapsed_time(end))
        took.append(min(times))
    assert max(took[1:]) < 3.5 * took[0], took


def test_tile_lists_that_are_not_valid_are_refused():
    for rows, cols in (([0, 5], [0, 0]), ([0, 0], [1, 1]), ([-1, 0], [0, 0])):
        br, bc = torch.tensor(rows, dtype=torch.int32, device="cuda"), torch.tensor(cols, dtype=torch.int32, device="cuda")
        a = void.VOIDTensor(torch.randn(2, 32, 32, device="cuda"), br, bc, torch.zeros(2, dtype=torch.int64, device="cuda"),
                            (64, 64), (32, 32), 0, 2, 0.5)
        b = torch.randn(64, 8, device="cuda")
        for call in (a.get_row_block_info, lambda: void.void_spmm(a, b), lambda: void.quantize_void_tensor(a).packed(),
                     lambda: void.void_tensor_to_fp8(a).packed_split(2)):
            with pytest.raises(ValueError, match="invalid VOID tile list"):
                call()


# ------------------------------------------------------------------------------------------ few columns
def _integer_matrix(m, k, density, seed):
    gen = torch.Generator().manual_seed(seed)
    nbr, nbc = (m + 31) // 32, (k + 31) // 32
    mask = torch.rand(nbr, nbc, generator=gen) < density
    mask[nbr // 2] = False                                                # an empty tile row
    mask[0, nbc - 1] = True
    dense = torch.randint(-3, 4, (m, k), generator=gen).float()
    return dense * mask.repeat_interleave(32, 0).repeat_interleave(32, 1)[:m, :k], gen


@pytest.mark.parametrize("dtype", [torch.int8, torch.float8_e4m3fn, torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m,k,density", [(32, 32, 1.0), (95, 200, 0.7), (330, 1100, 0.9), (64, 2500, 0.8)])
def test_products_with_few_columns_are_exact_on_small_integers(dtype, m, k, density):
    dense, gen = _integer_matrix(m, k, density, m + k)
    a = void.dense_to_void(dense.cuda())
    scale = 1.0
    if dtype == torch.int8:
        q = void.quantize_void_tensor(a)
        q.values, q.scales = a.values.to(torch.int8), torch.ones_like(q.scales)
    elif dtype == torch.float8_e4m3fn:
        q = void.void_tensor_to_fp8(a)
        q.values_fp8 = a.values.to(dtype)
        q.scaling_info.scale = torch.ones_like(q.scaling_info.scale)
    else:
        q = a.to_dtype(dtype)
    for n in (1, 2, 7, 8, 9, 16, 17, 31, 32, 33, 63, 64, 100, 128, 129):
        b = torch.randint(-3, 4, (k, n), generator=gen).float()
        ref = dense.double() @ b.double()
        bias = torch.randint(-4, 5, (n,), generator=gen).float()
        if dtype == torch.int8:
            cs = torch.tensor([1.0, 2.0, 0.5]).repeat(n)[:n]
            got = void.void_spmm_int8(q, b.to(torch.int8).cuda(), cs.cuda() if n > 1 else scale, bias=bias.cuda())
            assert torch.equal(got.double().cpu(), ref * (cs.double() if n > 1 else 1.0) + bias.double()), n
            y = void.void_linear(q, b.t().contiguous().to(torch.int8).cuda(), None, 1)
            assert torch.equal(y.double().cpu(), ref.t().clamp(min=0)), n
        elif dtype == torch.float8_e4m3fn:
            b8 = torch.zeros(k, (n + 15) // 16 * 16, dtype=torch.float8_e4m3fn, device="cuda")[:, :n]
            b8.view(torch.uint8).copy_(b.to(dtype).view(torch.uint8).cuda())
            got = void.void_spmm_fp8(q, b8, torch.float32, bias=bias.cuda())
            assert torch.equal(got.double().cpu(), ref + bias.double()), n
        else:
            bd = b.cuda().to(dtype)
            got = void.void_spmm(q, bd, bias=bias.cuda())
            assert torch.equal(got.double().cpu(), (ref + bias.double()).to(dtype).double()), n
            rb = torch.randint(-4, 5, (m,), generator=gen).float().cuda()
            y = void.void_linear(q, bd.t().contiguous(), rb)
            assert torch.equal(y.double().cpu(), (ref.t() + rb.double().cpu()).to(dtype).double()), n
    if dtype not in (torch.int8, torch.float8_e4m3fn):
        x = torch.randint(-3, 4, (k,), generator=gen).float()
        y = void.void_spmv(q, x.cuda().to(dtype))
        assert torch.equal(y.double().cpu(), (dense.double() @ x.double()).to(dtype).double())
        wide = torch.zeros(m, 3, dtype=dtype, device="cuda")
        void.void_spmv(q, x.cuda().to(dtype), wide[:, 1])                # a result with a stride
        assert torch.equal(wide[:, 1], y)
    void.check_device_status()


# ------------------------------------------------------------------------------------------ many tile rows
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m,k,n,density", [(3169, 1000, 300, 0.2), (9473, 330, 1100, 0.3), (4800, 1250, 260, 0.5), (2401, 640, 1030, 0.9)])
def test_products_with_many_tile_rows_are_exact_on_small_integers(dtype, m, k, n, density):
    dense, gen = _integer_matrix(m, k, density, m + k)
    a = void.dense_to_void(dense.cuda()).to_dtype(dtype)
    b = torch.randint(-3, 4, (k, n), generator=gen).float().cuda()
    ref = dense.cuda().double() @ b.double()
    bias = torch.randint(-4, 5, (n,), generator=gen).float().cuda()
    rb = torch.randint(-4, 5, (m,), generator=gen).float().cuda()
    for _ in range(3):
        got = void.void_spmm(a, b.to(dtype), bias=bias)
        assert torch.equal(got.double(), (ref + bias.double()).to(dtype).double())
        y = void.void_linear(a, b.to(dtype).t().contiguous(), rb, 1)
        assert torch.equal(y.double(), (ref.t() + rb.double()).clamp(min=0).to(dtype).double())
    void.check_device_status()


@pytest.mark.parametrize("dtype", [torch.int8, torch.float16, torch.float32])
@pytest.mark.parametrize("rows,cols,off", [(1, 1, 0), (3, 130, 1), (64, 64, 0), (129, 31, 0), (33, 257, 0), (200, 96, 2)])
def test_transposed_copies(dtype, rows, cols, off):
    from void_b200 import _lib
    es = torch.empty(0, dtype=dtype).element_size()
    x = torch.randint(-100, 100, (rows, cols + 3), device="cuda").to(dtype)[:, off:off + cols]
    ld = (rows * es + 15) // 16 * 16 // es
    out = torch.full((cols + 1, ld), 7, dtype=dtype, device="cuda")
    _lib.check(_lib.load().void_transpose(x.data_ptr(), x.stride(0) * es, out.data_ptr(), ld * es, es, rows, cols, _lib.stream_ptr(x.device)),
               "void_transpose")
    assert torch.equal(out[:cols, :rows], x.t()) and (out[:cols, rows:] == 0).all() and (out[cols] == 7).all()


@pytest.mark.parametrize("dtype", [torch.int8, torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m,k,n,density", [(4099, 2090, 1100, 0.85), (9000, 4100, 515, 0.5), (1030, 8200, 2050, 0.4)])
def test_large_linear_layers_are_exact_on_small_integers(dtype, m, k, n, density):
    dense, gen = _integer_matrix(m, k, density, m + k)
    a = void.dense_to_void(dense.cuda())
    x = torch.randint(-3, 4, (n, k), generator=gen).float().cuda()
    rb = torch.randint(-4, 5, (m,), generator=gen).float().cuda()
    ref = x.double() @ dense.cuda().double().t()
    if dtype == torch.int8:
        q = void.quantize_void_tensor(a)
        q.values, q.scales = a.values.to(torch.int8), torch.ones_like(q.scales)
        scale = torch.tensor([1.0, 2.0, 0.5]).repeat(n)[:n].cuda()
        for _ in range(2):
            y = void.void_linear(q, x.to(dtype), rb, x_scale=scale)
            assert torch.equal(y.double(), ref * scale.double()[:, None] + rb.double())
    else:
        a = a.to_dtype(dtype)
        wide = torch.zeros(n, k + 5, dtype=dtype, device="cuda")[:, 1:k + 1]      # rows off 16-byte boundaries
        wide.copy_(x)
        for b in (x.to(dtype), wide, wide):
            y = void.void_linear(a, b, rb, 1)
            assert torch.equal(y.double(), (ref + rb.double()).clamp(min=0).to(dtype).double())
        g = torch.randint(-2, 3, (n, m), generator=gen).float().cuda()
        layer = void.SparseLinear(k, m, a, bias=False)
        xg = x.to(dtype).requires_grad_(True)
        layer(xg).backward(g.to(dtype))
        assert torch.equal(xg.grad.double(), (g.double() @ dense.cuda().double()).to(dtype).double())
    void.check_device_status()


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m,k,n", [(64, 96, 1), (520, 330, 17), (4099, 1290, 129), (9001, 1100, 1500)])
def test_two_layers_are_exact_on_small_integers(dtype, m, k, n, density=0.3):
    d1, gen = _integer_matrix(m, k, density, m + k)
    d2, _ = _integer_matrix(k, m, density, m + n)
    w1, w2 = (void.dense_to_void(d.cuda()).to_dtype(dtype) for d in (d1, d2))
    x = torch.randint(-2, 3, (n, k), generator=gen).float().cuda()
    b1, b2 = (torch.randint(-4, 5, (s,), generator=gen).float().cuda() for s in (m, k))
    hidden = (x.double() @ d1.cuda().double().t() + b1.double()).clamp(min=0).to(dtype).double()
    ref = hidden @ d2.cuda().double().t() + b2.double()
    for _ in range(2):
        y = void.fused_sparse_mlp(x.to(dtype), w1, w2, "relu", b1, b2)
        assert y.dtype == dtype and torch.equal(y.double(), ref.to(dtype).double())
    void.check_device_status()


# ------------------------------------------------------------------------------------------ groups of tile rows
def test_two_layers_ask_the_interpreter_for_little_and_notice_every_change():
    """Calls the interpreter makes for a pass of two packed layers (17; 25 when every check was its own), and
    what such a pass must not overlook: edited and replaced weights, operands of another shape, type or length."""
    import sys
    gen = torch.Generator(device="cuda").manual_seed(2)
    layer = lambda m, k: void.dense_to_void(torch.randint(-2, 3, (m, k), generator=gen, device="cuda").half())
    w1, w2 = layer(128, 96), layer(64, 128)
    x = torch.randint(-2, 3, (8, 96), generator=gen, device="cuda").half()
    b1, b2 = (torch.randint(-2, 3, (m,), generator=gen, device="cuda").float() for m in (128, 64))

    def same(x, b1, b2):
        ref = (x.double() @ w1.to_dense().double().t() + (0 if b1 is None else b1.double())).clamp(min=0).to(x.dtype).double()
        ref = (ref @ w2.to_dense().double().t() + (0 if b2 is None else b2.double())).to(x.dtype)
        return torch.equal(void.fused_sparse_mlp(x, w1, w2, "relu", b1, b2), ref)

    assert same(x, b1, b2) and same(x, b1, b2) and same(x, None, b2) and same(x, b1, None)
    calls = [0]

    def count(frame, event, arg):
        calls[0] += event in ("call", "c_call")

    sys.setprofile(count)
    void.fused_sparse_mlp(x, w1, w2, "gelu", b1, b2)
    sys.setprofile(None)
    assert calls[0] <= 20, calls[0]
    w1.values[0, 0, 0] += 1                                                     # edited
    assert same(x, b1, b2)
    w2.values = w2.values * -1                                                  # replaced
    assert same(x, b1, b2) and same(x, b1, b2)
    assert same(x.reshape(2, 4, 96), b1, b2) and same(x[:, :].t().contiguous().t(), b1, b2)
    w32 = w1.to_dtype(torch.float32)                                            # types that differ
    assert torch.equal(void.fused_sparse_mlp(x, w32, w2, "none"), void.void_linear(w2, void.void_linear(w32, x)))
    with torch.inference_mode():                                                # nothing has a version: packed every time
        w1.values = w1.values * 1
        assert same(x, b1, b2)
        w1.values[0, 0, 1] += 1
        assert same(x, b1, b2)
    for bad in ((x[:, :64], b1, b2), (x, b1[:100], b2), (x, b1, b2[:32]), (x.cpu(), b1, b2)):
        with pytest.raises((AssertionError, RuntimeError, ValueError)):
            void.fused_sparse_mlp(bad[0], w1, w2, "relu", *bad[1:])
    void.check_device_status()


@pytest.mark.parametrize("kind,dtype,out", [("I8", torch.int8, torch.float32), ("I8", torch.int8, torch.float16),
                                            ("I8", torch.int8, torch.bfloat16), ("F16", torch.float16, torch.float16),
                                            ("BF16", torch.bfloat16, torch.bfloat16), ("TF32", torch.float32, torch.float32)])
@pytest.mark.parametrize("m,k,n,density,groups,entries,tiles", [
    (40, 70, 40, 0.9, 1, 1, 2), (250, 300, 129, 0.6, 1, 1, 8), (2500, 333, 384, 0.4, 12, 2, 8), (1111, 2000, 200, 0.95, 18, 1, 2),
    (10000, 640, 515, 0.1, 60, 2, 16)])
def test_grouped_products_are_exact_on_small_integers(kind, dtype, out, m, k, n, density, groups, entries, tiles):
    if dtype == torch.float32:                                            # (two stages have to fit a CTA's shared memory)
        entries, tiles = 1, ((m + 31) // 32 + groups - 1) // groups
    _grouped_exact(kind, dtype, out, m, k, n, density, groups, entries, tiles)


# Stages that end in the middle of a block column, runs of one to four rows, groups of two, five and eight rows, more groups than CTAs,
# and the stage shapes that products choose for 8 and 7 rows.
@pytest.mark.parametrize("kind,dtype,out,m,k,n,density,groups,entries,tiles", [
    ("I8", torch.int8, torch.float16, 256, 640, 130, 1.0, 1, 6, 2), ("I8", torch.int8, torch.float32, 2100, 900, 128, 0.5, 9, 6, 26),
    ("I8", torch.int8, torch.bfloat16, 500, 500, 77, 0.7, 8, 5, 14), ("BF16", torch.bfloat16, torch.bfloat16, 155, 700, 264, 0.8, 1, 3, 5),
    ("F16", torch.float16, torch.float16, 4800, 2100, 640, 0.15, 20, 3, 5), ("F16", torch.float16, torch.float16, 1000, 333, 512, 0.5, 4, 2, 1),
    ("TF32", torch.float32, torch.float32, 224, 640, 200, 0.6, 1, 1, 5), ("TF32", torch.float32, torch.float32, 2048, 1000, 384, 0.3, 8, 2, 5),
    ("TF32", torch.float32, torch.float16, 300, 700, 128, 0.9, 2, 2, 1)])
def test_grouped_stages_and_runs_are_exact_on_small_integers(kind, dtype, out, m, k, n, density, groups, entries, tiles):
    _grouped_exact(kind, dtype, out, m, k, n, density, groups, entries, tiles)


def _grouped_exact(kind, dtype, out, m, k, n, density, groups, entries, tiles):
    import ctypes
    from void_b200 import _lib, _spmm
    lib, kd = _lib.load(), getattr(_lib, "KIND_" + kind)
    dense, gen = _integer_matrix(m, k, density, m + n)
    a = void.dense_to_void(dense.cuda())
    vals = a.values.to(dtype)
    p = _spmm._mark_ready(_spmm.pack(vals, torch.ones(a.n_blocks, device="cuda") if kd == _lib.KIND_I8 else None, a.block_rows,
                                     a.block_cols, (m, k), kd))
    es, P = vals.element_size(), _lib.ptr
    ints = dict(dtype=torch.int32, device="cuda")
    rows, stages = torch.empty(groups * 16, **ints), torch.empty(groups + 1, **ints)
    records, ws = torch.empty(8 * p.nnz, **ints), torch.empty(2 * groups + p.nnz, **ints)
    blob = torch.empty(p.nnz * (1024 * es + 128), dtype=torch.uint8, device="cuda")
    _lib.check(lib.void_group_build(P(p.row_ptr), P(p.row_order), P(p.tile_cols), P(p.tiles), p.nbr, p.nnz, es, groups, entries,
                                    tiles, P(rows), P(stages), P(records), P(blob), P(ws), _lib.stream_ptr(blob.device)), "void_group_build")
    s = _lib.GroupStore(blob.data_ptr(), records.data_ptr(), stages.data_ptr(), rows.data_ptr(), groups, entries, tiles, 0)
    ld = (n * es + 15) // 16 * 16 // es
    b = torch.zeros(k, ld, dtype=dtype, device="cuda")[:, :n]
    x = torch.randint(-3, 4, (k, n), generator=gen).float().cuda()
    b.view(torch.uint8).copy_(x.to(dtype).view(torch.uint8)) if es == 1 else b.copy_(x)
    bias, rb = (torch.randint(-4, 5, (z,), generator=gen).float().cuda() for z in (n, m))
    ref = (dense.cuda().double() @ x.double() + bias.double() + rb.double()[:, None]).clamp(min=0).to(out)
    for tr in (0, 2):
        c = torch.empty(n, m, dtype=out, device="cuda") if tr else torch.empty(m, n, dtype=out, device="cuda")
        g = _lib.SpmmArgs()
        g.row_ptr, g.row_scale = p.row_ptr.data_ptr(), p.row_scale.data_ptr() if es == 1 else None
        g.nbr, g.nbc, g.nnz, g.tile_terms = p.nbr, p.nbc, p.nnz, 1
        g.b, g.ldb, g.K, g.N, g.b_scale = b.data_ptr(), ld * es, k, n, 1.0
        g.out, g.ldc, g.M, g.out_dtype, g.act, g.transposed = c.data_ptr(), c.stride(0), m, _lib.OUT_DTYPE_CODE[out], 1, tr
        g.bias, g.row_bias, g.status = bias.data_ptr(), rb.data_ptr(), _lib.status_word(c.device).data_ptr()
        _lib.check(lib.void_spmm_grouped(ctypes.byref(g), ctypes.byref(s), kd, _lib.stream_ptr(c.device)), "void_spmm_grouped")
        assert torch.equal(c.t() if tr else c, ref), tr
    void.check_device_status()


@pytest.mark.parametrize("dtype", [torch.int8, torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("m,k,density", [(9473, 700, 0.5), (5000, 1930, 0.9)])
def test_repeated_products_of_dense_tensors_stay_the_same(dtype, m, k, density):
    dense, gen = _integer_matrix(m, k, density, m + k)
    a = void.dense_to_void(dense.cuda())
    if dtype == torch.int8:
        q = void.quantize_void_tensor(a)
        q.values, q.scales = a.values.to(torch.int8), torch.ones_like(q.scales)
    else:
        q = a.to_dtype(dtype)
    for n in (1500, 520, 1030, 1500):
        x = torch.randint(-3, 4, (k, n), generator=gen).float().cuda()
        ref = dense.cuda().double() @ x.double()
        for _ in range(4):
            if dtype == torch.int8:
                assert torch.equal(void.void_spmm_int8(q, x.to(dtype), 1.0, out_dtype=torch.float32).double(), ref)
                y = void.void_linear(q, x.t().contiguous().to(dtype))
            else:
                assert torch.equal(void.void_spmm(q, x.to(dtype)).double(), ref.to(dtype).double())
                y = void.void_linear(q, x.t().contiguous().to(dtype))
            assert torch.equal(y.double(), ref.t().to(y.dtype).double())
    void.check_device_status()


@pytest.mark.parametrize("n", [224, 240, 241, 256, 257, 512, 513, 528, 529, 544])
def test_quantised_columns_around_the_widths_whose_grids_ask_for_more_shared_memory(n):
    b = torch.randn(700, n, generator=torch.Generator().manual_seed(n))
    q, s = void.quantize_cols_int8(b.cuda())
    ref_q, ref_s = vo.quantize_int8_cols(b.numpy())
    assert np.array_equal(s.cpu().numpy(), ref_s) and np.array_equal(q.cpu().numpy(), ref_q)
    f, fs, fi = void.quantize_cols_fp8(b.cuda())
    ref_f, ref_fs, ref_fi = vo.quantize_fp8_cols(b.numpy())
    assert np.array_equal(fs.cpu().numpy(), ref_fs) and np.array_equal(fi.cpu().numpy(), ref_fi)
    assert np.array_equal(f.view(torch.uint8).cpu().numpy(), ref_f)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("off", [0, 1, 3, 8])
def test_tiles_are_quantised_wherever_they_start(dtype, off):
    n = 5
    flat = torch.randn(n * 1024 + off, generator=torch.Generator().manual_seed(off)).to(dtype)
    values = flat.cuda()[off:].view(n, 32, 32)
    coords = torch.arange(n, dtype=torch.int32, device="cuda")
    a = void.VOIDTensor(values, coords, coords, torch.zeros(n, dtype=torch.int64, device="cuda"), (n * 32, n * 32), (32, 32), 0, n, 0.0)
    q = void.quantize_void_tensor(a)
    ref_q, ref_s = vo.quantize_int8_tiles(flat[off:].view(n, 32, 32).float().numpy())
    assert np.array_equal(q.values.cpu().numpy(), ref_q) and np.array_equal(q.scales.cpu().numpy(), ref_s)


# ------------------------------------------------------------------------------------------ passes over the columns of B
@pytest.mark.parametrize("dtype,k,n,linear", [
    ("int8", 65536, 512, False), ("int8", 65536, 600, False), ("int8", 65536, 1153, False), ("fp8", 65536, 641, False),
    (torch.bfloat16, 32768, 600, False), (torch.float16, 32768, 600, True), (torch.float32, 16384, 513, False),
    (torch.float32, 16384, 600, True)])
def test_products_in_passes_equal_products_of_few_columns(dtype, k, n, linear):
    """A B above three tenths of the L2 is multiplied in passes over its columns (the last one shorter), every product as in
    one of a few columns.  Small integers for the floating kinds, whose sums in any order are exact."""
    m, step, floating = 90, 256, isinstance(dtype, torch.dtype)
    gen = torch.Generator(device="cuda").manual_seed(k + n)
    mask = torch.rand(3, k // 32, generator=gen, device="cuda") < 0.05
    mask[1] = False
    numbers = lambda *size: (torch.randint(-2, 3, size, generator=gen, device="cuda").float() if floating
                             else torch.randn(*size, generator=gen, device="cuda"))
    a = void.void_from_block_mask(mask.cpu().numpy(), numbers(int(mask.sum()), 32, 32), shape=(m, k))
    a.values[a.block_rows == m // 32, m % 32:, :] = 0
    b = numbers(k, n)
    if dtype == "int8":
        q = void.quantize_void_tensor(a)
        bq, scale = void.quantize_cols_int8(b)
        product = lambda lo, hi: void.void_spmm_int8(q, bq[:, lo:hi], scale[lo:hi], out_dtype=torch.float16)
    elif dtype == "fp8":
        q = void.void_tensor_to_fp8(a)
        bq, scale = void.quantize_cols_fp8(b)[:2]
        product = lambda lo, hi: void.void_spmm_fp8(q, bq[:, lo:hi], torch.float16, b_scale=scale[lo:hi])
    elif linear:
        q, x = a.to_dtype(dtype), b.t().contiguous().to(dtype)
        product = lambda lo, hi: void.void_linear(q, x[lo:hi]).t()
    else:
        q, x = a.to_dtype(dtype), b.to(dtype)
        product = lambda lo, hi: void.void_spmm(q, x[:, lo:hi])
    whole = product(0, n)
    parts = [product(lo, min(n, lo + step)) for lo in range(0, n, step)]
    void.check_device_status()
    assert torch.equal(whole, torch.cat(parts, 1))


# ------------------------------------------------------------------------------------------ panels per item and CTA shapes
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("m,k,n,density,linear", [
    (2110, 300, 5700, 0.95, False),     # two panels per item (16 bits), an odd number of them
    (2080, 300, 5633, 0.7, False),      # rows too short for it
    (4250, 300, 5800, 0.95, True),      # two panels per item, x as it lies
    (2110, 640, 5700, 0.95, True),      # ... with fewer items and longer rows
    (16390, 640, 1100, 0.95, True),     # ... and x transposed first
    (9000, 300, 515, 0.5, True)])       # one panel, slim CTAs for every type
def test_large_floating_products_are_exact_on_small_integers(dtype, m, k, n, density, linear):
    dense, gen = _integer_matrix(m, k, density, m + n)
    a = void.dense_to_void(dense.cuda()).to_dtype(dtype)
    b = torch.randint(-2, 3, (n, k) if linear else (k, n), generator=gen).cuda().to(dtype)
    ref = b.double() @ dense.cuda().double().t() if linear else dense.cuda().double() @ b.double()
    for _ in range(2):
        y = void.void_linear(a, b) if linear else void.void_spmm(a, b)
        assert torch.equal(y.double(), ref.to(dtype).double())
    void.check_device_status()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m,k,n,density,linear", [
    (94720, 96, 128, 0.9, False), (94721, 96, 65, 0.9, False),                # one panel in all
    (31580, 300, 384, 0.7, False), (31580, 130, 257, 0.9, False),             # three: one per item, mid and slim CTAs
    (18950, 300, 640, 0.7, False), (18950, 130, 515, 0.9, False),             # five: one, and two with short rows
    (31580, 640, 384, 0.95, True), (10530, 300, 1152, 0.7, False)])           # three, transposed; nine: two
def test_products_with_an_odd_number_of_panels_are_exact_on_small_integers(dtype, m, k, n, density, linear):
    dense, gen = _integer_matrix(m, k, density, m + n)
    a = void.dense_to_void(dense.cuda()).to_dtype(dtype)
    b = torch.randint(-2, 3, (n, k) if linear else (k, n), generator=gen).cuda().to(dtype)
    ref = b.double() @ dense.cuda().double().t() if linear else dense.cuda().double() @ b.double()
    y = void.void_linear(a, b) if linear else void.void_spmm(a, b)
    assert torch.equal(y.double(), ref.to(dtype).double())
    void.check_device_status()


@pytest.mark.parametrize("m,k,n,density,linear", [(131072, 1024, 128, 0.3, False), (32768, 2048, 384, 0.2, False), (131072, 2048, 64, 0.3, True)])
def test_items_of_two_panels_are_no_slower_than_items_of_one(m, k, n, density, linear):
    """Where the launch chooses the panels per item (43, 18 and 29 % over the better shape of one panel when an item of two was
    half empty)."""
    from void_b200 import _lib, _spmm
    from void_b200.ops import packed_fp
    gen = torch.Generator(device="cuda").manual_seed(n)
    mask = torch.rand(m // 32, k // 32, generator=gen, device="cuda") < density
    a = void.void_from_block_mask(mask.cpu().numpy(), torch.randn(int(mask.sum()), 32, 32, generator=gen, device="cuda"), shape=(m, k)).to_dtype(torch.float16)
    p = packed_fp(a, _lib.FP_KIND[torch.float16])
    b = torch.randn((n, k) if linear else (k, n), generator=gen, device="cuda").half()
    out = torch.empty((n, m) if linear else (m, n), dtype=torch.float16, device="cuda")

    def time_of(**options):
        stream, times = torch.cuda.Stream(), []
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            for _ in range(8):
                _spmm.spmm(p, b, out, scale_mode=_lib.SCALE_ROW_MEAN, transposed=linear, **options)
        for _ in range(8):
            begin, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            begin.record()
            graph.replay()
            end.record()
            end.synchronize()
            times.append(begin.elapsed_time(end))
        return min(times)

    one = min(time_of(panels_per_item=1, cta_shape=shape) for shape in (1, 2, 6))
    assert time_of() < 1.1 * one


# ------------------------------------------------------------------------------------------ products behind what prepares B
@pytest.mark.parametrize("dtype,k,n", [
    (torch.bfloat16, 6880, 333), (torch.bfloat16, 6912, 333), (torch.float32, 64, 33),     # row copies: 1183, 1188 and 3 blocks
    ("int8", 512, 16), ("int8", 4096, 528), ("int8", 4096, 544), ("fp8", 2080, 528), ("fp8", 2080, 529)])   # 1, 33 and 34 clusters
def test_products_wait_for_the_kernel_that_prepares_their_operand(dtype, k, n):
    """The product's launch starts beside a kernel that copies or quantises B.  New values in the same buffers every time, so
    that a product which read too early would use those of the time before."""
    gen = torch.Generator(device="cuda").manual_seed(k + n)
    nbc = (k + 31) // 32
    mask = torch.rand(5, nbc, generator=gen, device="cuda") < 0.3
    mask[:, nbc - 1] = True
    values = torch.randint(-2, 3, (int(mask.sum()), 32, 32), generator=gen, device="cuda").float()
    a = void.void_from_block_mask(mask.cpu().numpy(), values, shape=(160, nbc * 32))
    q = {"int8": void.quantize_void_tensor, "fp8": void.void_tensor_to_fp8}.get(dtype, lambda t: t.to_dtype(dtype))(a)
    quantise = {"int8": void.quantize_cols_int8, "fp8": void.quantize_cols_fp8}.get(dtype)

    def product(b):
        if quantise is None:
            return void.void_spmm(q, b)
        c, scale = quantise(b)[:2]
        if dtype == "int8":
            return void.void_spmm_int8(q, c, scale, out_dtype=torch.float32)
        return void.void_spmm_fp8(q, c, torch.float32, b_scale=scale)

    inputs = [torch.randint(-4, 5, (nbc * 32, n), generator=gen, device="cuda").float() * 2.0 ** i for i in range(6)]
    if quantise is None:
        inputs = [b.to(dtype) for b in inputs]
    for b in inputs:
        product(b)                      # plans and stores are built
    torch.cuda.synchronize()
    for b, c in zip(inputs, [product(b) for b in inputs]):
        if quantise is None:
            ref = a.to_dense().double() @ b.double()
            assert torch.equal(c.double(), ref.to(dtype).double())
        else:
            x, scale = quantise(b)[:2]
            torch.cuda.synchronize()
            alone = (void.void_spmm_int8(q, x, scale, out_dtype=torch.float32) if dtype == "int8"
                     else void.void_spmm_fp8(q, x, torch.float32, b_scale=scale))
            assert torch.equal(c, alone)
    void.check_device_status()


@pytest.mark.parametrize("kind", ["int8", "fp8"])
@pytest.mark.parametrize("rows,k,n", [(592, 96, 128), (593, 96, 128), (148, 1312, 512), (149, 1312, 512), (1, 64, 40), (3, 4000, 136), (37, 700, 2000)])
def test_results_staged_in_the_ring_are_those_stored_directly(kind, rows, k, n):
    """One item per CTA up to 592 items (the staging tile then lies in the ring), more from there on; empty rows, ragged edges."""
    from void_b200 import _lib, _spmm
    gen = torch.Generator().manual_seed(rows + n)
    dense = torch.randn(rows * 32 - 5, k, generator=gen)
    keep = torch.rand(rows, (k + 31) // 32, generator=gen) < 0.4
    keep[rows // 2] = False                                              # an empty row of tiles
    keep[0] = True
    dense *= keep.repeat_interleave(32, 0).repeat_interleave(32, 1)[:dense.shape[0], :k]
    a = void.dense_to_void(dense.cuda())
    b = torch.randn(k, n, generator=gen).cuda()
    if kind == "int8":
        t = void.quantize_void_tensor(a)
        p, (q, scale) = t.packed(), void.quantize_cols_int8(b)
    else:
        t = void.void_tensor_to_fp8(a)
        p, (q, scale) = t.packed_split(2), void.quantize_cols_fp8(b)[:2]
        q = q.view(torch.uint8)
    bias = torch.randn(n, generator=gen).cuda()
    for dtype in (torch.float16, torch.bfloat16):
        outs = []
        for options in ({}, {"flags": 2}, {"grid": 5}):
            out = torch.full((dense.shape[0], n), float("nan"), dtype=dtype, device="cuda")
            _spmm.spmm(p, q, out, scale_mode=_lib.SCALE_ROW_MEAN, col_scale=scale, bias=bias, act=2, cta_shape=2, **options)
            outs.append(out)
        assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    void.check_device_status()


@pytest.mark.parametrize("kind,stages", [("int8", 2), ("int8", 3), ("int8", 9), ("int8", 10), ("int8", 14), ("fp8", 2), ("fp8", 12), ("fp8", 13), ("fp8", 16)])
def test_rings_of_as_many_ordinary_stages_as_are_asked_for(kind, stages):
    """One item per CTA, three CTAs per SM and 16-bit results: 14 stages of three INT8 units, 16 of two FP8 units of two terms fit a
    CTA's shared memory."""
    from void_b200 import _lib, _spmm, workloads
    w = workloads.block_sparse(workloads.uniform_mask(110, 40, 0.4, seed=stages), 384, seed=stages)
    if kind == "int8":
        p, (b, scale) = void.quantize_void_tensor(w.a).packed(), void.quantize_cols_int8(w.b)
    else:
        p, (b, scale) = void.void_tensor_to_fp8(w.a).packed_split(2), void.quantize_cols_fp8(w.b)[:2]
    outs = []
    for s in (0, stages):
        outs.append(torch.full((3520, 384), 7.0, dtype=torch.float16, device="cuda"))
        _spmm.spmm(p, b, outs[-1], scale_mode=_lib.SCALE_ROW_MEAN, col_scale=scale, panels_per_item=1, stages=s)
    assert torch.equal(*outs)
    void.check_device_status()


@pytest.mark.parametrize("dtype", [torch.int8, torch.float16, torch.float32])
def test_a_group_store_takes_what_its_kernels_use(dtype):
    """Tiles, 32 bytes of heads and a record of 32 bytes each; what belongs to groups and rows is within the slack."""
    from void_b200 import _lib, ops, workloads
    w = workloads.block_sparse(workloads.uniform_mask(157, 61, 0.1, seed=3), 1500, seed=3)
    if dtype == torch.int8:
        a, (b, scale) = void.quantize_void_tensor(w.a), void.quantize_cols_int8(w.b)
        product, packed = lambda: void.void_spmm_int8(a, b, scale), lambda: a.packed()
    else:
        a, b = w.a.to_dtype(dtype), w.b.to(dtype)
        product, packed = lambda: void.void_spmm(a, b), lambda: ops.packed_fp(a, ops.product_kind(a, b))
    for _ in range(4):
        product()
        torch.cuda.synchronize()
    assert _lib.native().packed_grouped(packed().native, None)[1] == 1
    requested = lambda: torch.cuda.memory_stats()["requested_bytes.all.current"]
    before = requested()
    void.allow_group_stores(a, False)
    assert 0 < before - requested() - a.n_blocks * 1024 * a.values.element_size() <= a.n_blocks * 64 + 32768


@pytest.mark.parametrize("es", [1, 2, 4])
def test_a_group_store_is_written_inside_its_blob(es):
    """Every tile a stage of its own, so that there are as many heads as there can be."""
    from void_b200 import _lib
    lib, P = _lib.load(), _lib.ptr
    nbr, nbc, groups = 24, 37, 3
    nnz, ints = nbr * nbc, dict(dtype=torch.int32, device="cuda")
    row_ptr, cols = torch.arange(0, nnz + 1, nbc, **ints), torch.arange(nbc, **ints).repeat(nbr)
    tiles = torch.randint(0, 255, (nnz * 1024 * es,), dtype=torch.uint8, device="cuda")
    rows, stages, records, ws = (torch.zeros(n, **ints) for n in (groups * 16, groups + 1, 8 * nnz, 2 * groups + nnz))
    size = nnz * (1024 * es + 32)
    blob = torch.full((size + 4096,), 0xa5, dtype=torch.uint8, device="cuda")
    _lib.check(lib.void_group_build(P(row_ptr), None, P(cols), P(tiles), nbr, nnz, es, groups, 1, 1, P(rows), P(stages), P(records), P(blob),
                                    P(ws), _lib.stream_ptr(blob.device)), "void_group_build")
    assert stages.tolist() == [0, nnz // 3, 2 * nnz // 3, nnz] and bool((blob[size:] == 0xa5).all())
    place = ws[2 * groups:].long()
    assert torch.equal(blob[:nnz * 1024 * es].view(nnz, -1)[place], tiles.view(nnz, -1))
    heads = blob[nnz * 1024 * es:size].view(2, nnz, 16)
    assert torch.equal(heads[:, :, 1].sum(0), torch.ones(nnz, dtype=torch.int64, device="cuda"))     # one run in all per stage
