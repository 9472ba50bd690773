"""The penalty kernel against the tensor operations it stands in for.

Both are evaluated on the same image; the operations in 64 bits are the
reference.  float64 results agree to the rounding of sums of at most 26
terms per voxel (gradient, 1e-13 of its largest value) and of 1e6 terms
(value, 1e-12); the float32 gradient is the 64-bit one rounded once (1.2e-7 of
its value, and of the largest).
"""
import pytest
import torch

from fir_b200 import autograd as fa

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 1, 7), (2, 1, 5, 4), (3, 2, 2, 2), (2, 33, 17, 9), (64, 65, 66)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("contiguous", [True, False])
def test_value_and_gradient(shape, dtype, contiguous):
    gen = torch.Generator(device="cuda").manual_seed(3)
    x = torch.rand(shape, generator=gen, device="cuda", dtype=dtype) * 3
    if not contiguous:
        x = x.transpose(-1, -2)
    ref = x.double().detach().requires_grad_(True)
    want = fa._penalty_of_pairs(ref, 0.3)
    want_g, = torch.autograd.grad(2.5 * want, ref) if want.requires_grad and want != 0 else (torch.zeros_like(ref),)
    x = x.detach().requires_grad_(True)
    assert fa._plain_cuda_image(x, 0.3)
    got = fa.quadratic_penalty(x, 0.3)
    assert got.dtype == dtype and got.shape == ()
    (2.5 * got).backward()
    assert x.grad.dtype == dtype and x.grad.shape == x.shape
    rel = 1e-12 if dtype == torch.float64 else 1.2e-7
    assert abs(float(got.detach()) - float(want.detach())) <= rel * abs(float(want.detach()))
    top = float(want_g.abs().max())
    tol = 1e-13 * top if dtype == torch.float64 else 2.4e-7 * top
    assert float((x.grad.double() - want_g).abs().max()) <= tol


def test_second_derivative_and_transforms_use_the_operations():
    gen = torch.Generator(device="cuda").manual_seed(4)
    x = torch.rand((5, 6, 7), generator=gen, device="cuda", dtype=torch.float64).requires_grad_(True)
    v = torch.rand(x.shape, generator=gen, device="cuda", dtype=torch.float64)
    g, = torch.autograd.grad(fa.quadratic_penalty(x, 0.7), x, create_graph=True)
    hv, = torch.autograd.grad((g * v).sum(), x)
    want, = torch.autograd.grad(fa._penalty_of_pairs(v.requires_grad_(True), 0.7), v)  # quadratic: H v = grad at v
    assert torch.allclose(hv, want, rtol=1e-12, atol=1e-12)
    v = v.detach()
    out, tangent = torch.func.jvp(lambda t: fa.quadratic_penalty(t, 0.7), (x.detach(),), (v,))
    assert torch.allclose(tangent, (g.detach() * v).sum(), rtol=1e-12)
    per = torch.func.vmap(lambda t: fa.quadratic_penalty(t, 0.7))(torch.stack([x.detach(), v]))
    assert torch.allclose(per[1], fa.quadratic_penalty(v, 0.7), rtol=1e-12)
    with torch.autograd.forward_ad.dual_level():
        dual = torch.autograd.forward_ad.make_dual(x.detach(), v)
        t = torch.autograd.forward_ad.unpack_dual(fa.quadratic_penalty(dual, 0.7)).tangent
    assert torch.allclose(t, tangent, rtol=1e-12)
