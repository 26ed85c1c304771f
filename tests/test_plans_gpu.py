"""Work plans of power-law products: which tile list they were made for, and how long graphs may read them."""
import pytest
import torch

import void_b200 as void
from void_b200 import workloads

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
