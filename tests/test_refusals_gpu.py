"""Operands that are shorter than what a kernel reads or writes are refused on the host, before any launch."""
import pytest
import torch

import void_b200 as void
from void_b200 import _spmm, stream_k, workloads

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def case():
    w = workloads.block_sparse(workloads.uniform_mask(6, 5, 0.5, seed=1), 40, seed=1)
    return w, void.quantize_void_tensor(w.a), void.void_tensor_to_fp8(w.a), void.quantize_cols_int8(w.b), void.quantize_cols_fp8(w.b)


def test_short_column_scales_and_biases(case):
    w, q, f, (bq, bs), (bf, fs, _) = case
    short, long_ = torch.ones(39, device="cuda"), torch.ones(41, device="cuda")
    x = bq.t().contiguous()
    for call in (lambda v: void.void_spmm_int8(q, bq, bs, bias=v), lambda v: void.void_linear(q, x, x_scale=v),
                 lambda v: void.void_spmm_fp8(f, bf, b_scale=v), lambda v: void.void_spmm_fp8(f, bf, b_scale=fs, bias=v),
                 lambda v: void.void_spmm_fp8(f, bf, b_scale=v, scale_terms=0), lambda v: void.void_spmm(w.a, w.b, bias=v),
                 lambda v: void.void_spmm_stream_k(q, bq, b_scale=bs, bias=v)):
        with pytest.raises(void.VoidB200Error, match="must have 40 elements, got 39"):
            call(short)
        assert torch.equal(call(long_), call(long_[:40]))              # what lies behind the last column is not read
    void.check_device_status()


def test_short_arrays_for_raw_sums(case):
    w, q, _, (bq, bs), _ = case
    acc = torch.zeros(6 * 32 * 40, dtype=torch.int32, device="cuda")
    assert void.void_spmm_int8(q, bq, bs, acc_out=acc).shape == (192, 40)
    for bad in (acc[:-1], acc.to(torch.int64), acc.cpu(), acc.reshape(40, -1).t()):
        with pytest.raises(void.VoidB200Error):
            void.void_spmm_int8(q, bq, bs, acc_out=bad)
    wl = void.compute_stream_k_workload(q, 8, 4)
    plan = stream_k.stream_k_plan(q, 40, wl, per_worker=True, n_cta=8)
    parts = torch.zeros(plan.n_segs, 32, 40, dtype=torch.int32, device="cuda")
    void.void_spmm_stream_k(q, bq, wl, b_scale=bs, worker_partials=parts, n_cta=8)
    with pytest.raises(void.VoidB200Error, match="worker_partials"):
        void.void_spmm_stream_k(q, bq, wl, b_scale=bs, worker_partials=parts[:-1], n_cta=8)
    void.check_device_status()


def test_lists_and_values_of_different_lengths(case):
    w, q, f, (bq, bs), _ = case
    a, n = w.a, w.a.n_blocks

    def tensor(values=a.values, rows=a.block_rows, cols=a.block_cols):
        return void.VOIDTensor(values, rows, cols, a.morton_codes, a.shape, (32, 32), 0, n, 0.0)

    for t in (tensor(rows=a.block_rows[:-1], cols=a.block_cols[:-1]), tensor(values=a.values[:-1]), tensor(cols=a.block_cols[:-1])):
        for call in (lambda: void.void_spmm(t, w.b), lambda: void.quantize_void_tensor(t).packed(),
                     lambda: void.void_tensor_to_fp8(t).packed(), lambda: void.void_tensor_to_fp8(t).packed_split(2)):
            with pytest.raises(ValueError, match="invalid VOID tile list"):
                call()
    with pytest.raises(ValueError, match="invalid VOID tile list"):
        tensor(cols=a.block_cols[:-1]).get_row_block_info()
    row_ptr, block_indices = a.get_row_block_info()
    for rp, bi in ((row_ptr[:-1], block_indices), (row_ptr, block_indices[:-1]), (row_ptr, block_indices.long())):
        with pytest.raises(ValueError, match="invalid VOID tile index"):
            _spmm.pack(a.values, None, a.block_rows, a.block_cols, a.shape, 4, rp, bi)


def test_values_that_do_not_belong_to_the_layer(case):
    w = case[0]
    a, x = w.a, w.b.t().contiguous()
    for values, count in ((a.values[:-1], a.n_blocks), (a.values.reshape(-1, 16, 64), a.n_blocks)):
        with pytest.raises(void.VoidB200Error, match="tiles of 32x32"):
            void.VOIDLinearFunction.apply(values, a.block_rows, a.block_cols, a.shape, (32, 32), count, x, None)
    with pytest.raises(ValueError, match="invalid VOID tile index"):
        void.VOIDLinearFunction.apply(a.values, a.block_rows, a.block_cols, a.shape, (32, 32), a.n_blocks + 1, x, None)
    void.check_device_status()
