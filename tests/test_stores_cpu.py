"""What says whether a store, an index or a plan derived from a tensor's fields still belongs to them."""
import torch

from void_b200 import _lib


def test_identity_follows_contents_layout_and_storage():
    native = _lib.native()
    a, b = torch.zeros(4, 8), torch.arange(6)
    known = native.identity(a, None, b)
    assert native.unchanged(known, a, None, b) and native.unchanged(known, a.detach(), None, b.view(6))
    assert not native.unchanged(known, a, b, b) and not native.unchanged(known, a, None, None)
    assert not native.unchanged(known, a.t(), None, b)                          # the same memory read another way
    assert not native.unchanged(known, a[:2], None, b)
    assert not native.unchanged(known, a.view(torch.int32), None, b)
    assert not native.unchanged(known, a.clone(), None, b)
    b[::2] = 1
    assert not native.unchanged(known, a, None, b)


def test_identity_of_a_dropped_tensor_is_never_met_again():
    native = _lib.native()
    for nbytes in (64, 4096, 1 << 20):
        t = torch.zeros(nbytes, dtype=torch.uint8)
        ptr, known = t.data_ptr(), native.identity(t)
        del t
        again = [torch.zeros(nbytes, dtype=torch.uint8) for _ in range(64)]     # one of them usually lies at the same address
        assert not any(native.unchanged(known, x) for x in again), ptr in {x.data_ptr() for x in again}


def test_inference_tensors_are_taken_as_changed():
    with torch.inference_mode():
        t = torch.zeros(8)
        known = _lib.native().identity(t)
        t.add_(1)                                                               # leaves no trace
        assert not _lib.native().unchanged(known, t)
