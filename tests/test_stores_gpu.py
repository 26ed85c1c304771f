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
