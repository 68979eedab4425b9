"""Backward of the fused losses in the forms where the scaled gradients are more than two products
of plain tensors: a loss gradient that carries a tangent, and saved-tensor hooks that give the saved
gradients back as conjugate or negative views."""

import pytest
import torch
from torch.autograd import forward_ad

pytestmark = pytest.mark.gpu


def problem():
    from ptychox_b200 import ptychoX_base_loss

    gen = torch.Generator(device="cuda").manual_seed(8)
    obj = torch.randn(48, 48, dtype=torch.complex64, generator=gen, device="cuda", requires_grad=True)
    probe = torch.randn(16, 16, dtype=torch.complex64, generator=gen, device="cuda", requires_grad=True)
    pos = torch.tensor([[0, 0], [20, 9], [32, 32]], device="cuda")
    counts = torch.randint(0, 50, (3, 16, 16), generator=gen, device="cuda").to(torch.int32).to(torch.uint16)
    return obj, probe, lambda: ptychoX_base_loss(obj, probe, pos, counts, 0.5)


def close(got, want, factor=1.0):
    """Float2 atomics order the sums of the sweep, so to FP32 rounding of them."""
    for a, b in zip(got, want):
        assert torch.linalg.norm(a - factor * b) <= 1e-6 * abs(factor) * torch.linalg.norm(b)


def test_a_tangent_of_the_loss_gradient_reaches_the_gradients():
    obj, probe, loss = problem()
    want = torch.autograd.grad(loss(), (obj, probe))
    value = loss()
    with forward_ad.dual_level():
        seed = forward_ad.make_dual(torch.tensor(2.0, dtype=torch.float64, device="cuda"),
                                    torch.tensor(-3.0, dtype=torch.float64, device="cuda"))
        dual = [forward_ad.unpack_dual(g) for g in torch.autograd.grad(value, (obj, probe), grad_outputs=seed)]
        assert all(d.tangent is not None for d in dual)
        close([d.primal for d in dual], want, 2.0)
        close([d.tangent for d in dual], want, -3.0)


@pytest.mark.parametrize("pack, unpack", [
    (lambda t: t.conj().resolve_conj(), lambda t: t.conj()),
    (lambda t: -t, lambda t: torch._neg_view(t)),
])
def test_views_from_saved_tensor_hooks(pack, unpack):
    obj, probe, loss = problem()
    want = torch.autograd.grad(loss(), (obj, probe))
    with torch.autograd.graph.saved_tensors_hooks(lambda t: pack(t.detach()), unpack):
        value = loss()
    close(torch.autograd.grad(value, (obj, probe)), want)
