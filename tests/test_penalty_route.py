"""CPU tests of the choice between the penalty's kernel and its tensor
operations (the tensors' ``is_cuda`` is replaced; no GPU call is made)."""
import pytest
import torch

from fir_b200 import autograd


@pytest.fixture
def claims_cuda(monkeypatch):
    monkeypatch.setattr(torch.Tensor, "is_cuda", property(lambda self: True))


PRIVATE = [(torch._C._functorch, "peek_interpreter_stack"), (torch._C._functorch, "is_functorch_wrapped_tensor"),
           (torch.autograd.forward_ad, "_current_level"), (torch._C, "_len_torch_dispatch_stack"),
           (torch._C, "_len_torch_function_stack")]


@pytest.mark.parametrize("holder,name", PRIVATE, ids=[n for _, n in PRIVATE])
def test_a_torch_without_its_private_names_takes_the_operations(claims_cuda, monkeypatch, holder, name):
    x = torch.rand(2, 3, 4, dtype=torch.float64)
    want = autograd._penalty_of_pairs(x, 0.5)
    assert autograd._plain_cuda_image(x, 0.5)
    monkeypatch.delattr(holder, name)
    assert not autograd._plain_cuda_image(x, 0.5)
    assert torch.equal(autograd.quadratic_penalty(x, 0.5), want)


def test_a_negated_view_takes_the_operations(claims_cuda):
    """Its memory holds the other signs, and contiguous() leaves it so."""
    x = torch._neg_view(torch.rand(2, 3, 4))
    assert x.contiguous().data_ptr() == x.data_ptr()
    assert not autograd._plain_cuda_image(x, 0.5)
    assert autograd._plain_cuda_image(x.resolve_neg(), 0.5)
