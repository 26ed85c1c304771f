"""The autograd node of the sparse product beside the rest of the autograd engine: saved-tensor hooks, checkpoints, versions,
retained and recorded backward passes, and the derivatives it does not have."""
import pytest
import torch
from torch.utils.checkpoint import checkpoint

import void_b200 as void
from void_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.fixture()
def layer_and_input():
    w = workloads.block_sparse(workloads.uniform_mask(5, 7, 0.5, seed=1), 8, seed=1)
    lin = void.SparseLinear(224, 160, w.a, bias=True)
    gen = torch.Generator(device="cuda").manual_seed(1)
    with torch.no_grad():
        lin.bias.copy_(torch.randn(160, device="cuda", generator=gen))
    return lin, torch.randn(50, 224, device="cuda", generator=gen, requires_grad=True)


def _grads(lin, x, run):
    for p in (*lin.parameters(), x):
        p.grad = None
    y = run(x)
    (y * y).sum().backward()
    return [y.detach()] + [p.grad.clone() for p in (*lin.parameters(), x)]


@pytest.mark.parametrize("reentrant", [True, False])
def test_checkpoints_around_the_layer_and_around_what_it_reads(layer_and_input, reentrant):
    lin, x = layer_and_input
    plain = lambda t: lin(torch.tanh(t * 2))
    want = _grads(lin, x, plain)
    for run in (lambda t: checkpoint(plain, t, use_reentrant=reentrant),
                lambda t: lin(checkpoint(lambda u: torch.tanh(u * 2), t, use_reentrant=reentrant)),
                lambda t: checkpoint(lambda u: lin(checkpoint(lambda z: torch.tanh(z * 2), u, use_reentrant=False)), t,
                                     use_reentrant=reentrant)):
        for a, b in zip(_grads(lin, x, run), want):
            assert torch.equal(a, b)
    void.check_device_status()


def test_hooks_on_saved_tensors_run_with_autograd_on(layer_and_input):
    lin, x = layer_and_input
    want = _grads(lin, x, lin)
    recorded = []

    def unpack(t):
        with torch.enable_grad():                       # what a checkpoint does: a forward pass of its own
            z = torch.ones(3, device="cuda", requires_grad=True)
            recorded.append((z * 2).grad_fn is not None)
        return t.cuda()

    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.cpu(), unpack):
        got = _grads(lin, x, lin)
    assert len(recorded) >= 2 and all(recorded)
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    with torch.autograd.graph.save_on_cpu():
        for a, b in zip(_grads(lin, x, lin), want):
            assert torch.equal(a, b)


def test_versions_and_freed_buffers(layer_and_input):
    lin, x = layer_and_input
    y = lin(x).sum()
    y.backward(retain_graph=True)
    first = x.grad.clone()
    y.backward()
    assert torch.equal(x.grad, 2 * first)
    with pytest.raises(RuntimeError, match="second time"):
        y.backward()
    y = lin(x).sum()
    with torch.no_grad():
        lin.sparse_weight.values.mul_(2)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.backward()


def test_a_recorded_backward_pass_keeps_the_bias_gradient_differentiable(layer_and_input):
    lin, x = layer_and_input
    y = lin(x.detach())
    scale = torch.full((), 3.0, device="cuda", requires_grad=True)
    (gb,) = torch.autograd.grad((y * scale).sum(), lin.bias, create_graph=True)
    (gs,) = torch.autograd.grad(gb.sum(), scale)        # d/ds sum over (rows, columns) of s
    assert float(gs) == 50 * 160


def test_derivatives_that_there_are_not_are_refused(layer_and_input):
    import torch.autograd.forward_ad as fwad
    lin, x = layer_and_input
    with fwad.dual_level():
        with pytest.raises(NotImplementedError, match="forward-mode"):
            lin(fwad.make_dual(x.detach(), torch.ones_like(x)))
    v = lin.sparse_weight.values.detach()
    a = lin.sparse_weight.get_void_tensor()
    call = lambda values, t: void.VOIDLinearFunction.apply(values, a.block_rows, a.block_cols, a.shape, (32, 32), a.n_blocks, t, None)
    for transform in (lambda: torch.func.grad(lambda t: call(v, t).sum())(x.detach()),
                      lambda: torch.func.vmap(lambda t: call(v, t))(x.detach()[None]),
                      lambda: torch.func.jvp(lambda t: call(v, t), (x.detach(),), (x.detach(),))):
        with pytest.raises(RuntimeError, match="torch.func"):
            transform()
