"""Backward of the fused losses: the saved unit-loss gradients times the loss gradient in one
launch (``ptx_scale_gradients``), against torch's products, and the backward forms that take those
products themselves."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(0, 3), (1, 1), (2, 7), (1023, 1024), (4097, 70001)])
@pytest.mark.parametrize("offset", [0, 1])
def test_scaled_gradients_equal_the_products(sizes, offset):
    """Even and odd lengths, arrays on and 8 bytes off a 16-byte boundary, finite and not: the
    same single rounding per part, so the values are equal."""
    from ptychox_b200 import _abi
    from ptychox_b200._utils import call_on

    gen = torch.Generator(device="cuda").manual_seed(sizes[0] + offset)
    arrays = [torch.randn(n + offset, dtype=torch.complex64, generator=gen, device="cuda")[offset:] for n in sizes]
    if sizes[0] > 4:
        arrays[0][3] = complex(float("inf"), 1.0)
        arrays[0][4] = complex(0.0, float("nan"))
    g = torch.tensor(-0.37, dtype=torch.float64, device="cuda")
    outs = [torch.empty(n + offset, dtype=torch.complex64, device="cuda")[offset:] for n in sizes]
    call_on(torch.device("cuda", torch.cuda.current_device()), "ptx_scale_gradients", g.data_ptr(),
            arrays[0].data_ptr(), outs[0].data_ptr(), sizes[0], arrays[1].data_ptr(), outs[1].data_ptr(), sizes[1])
    for a, o in zip(arrays, outs):
        want = torch.view_as_real(a * g.to(torch.float32))
        assert torch.equal(torch.nan_to_num(torch.view_as_real(o)), torch.nan_to_num(want))
    with pytest.raises(ValueError):
        _abi.call("ptx_scale_gradients", None, None, None, 0, None, None, 0, 0)


def problem():
    from ptychox_b200 import ptychoX_base_loss

    gen = torch.Generator(device="cuda").manual_seed(5)
    obj = torch.randn(48, 48, dtype=torch.complex64, generator=gen, device="cuda", requires_grad=True)
    probe = torch.randn(16, 16, dtype=torch.complex64, generator=gen, device="cuda", requires_grad=True)
    pos = torch.tensor([[0, 0], [20, 9], [32, 32]], device="cuda")
    counts = torch.randint(0, 50, (3, 16, 16), generator=gen, device="cuda").to(torch.int32).to(torch.uint16)
    return obj, probe, lambda: ptychoX_base_loss(obj, probe, pos, counts, 0.5)


def test_backward_forms_agree():
    """Plain, retained, with create_graph, batched over loss gradients, and through hooks that
    move saved tensors to the host; float2 atomics order the sums, so to FP32 rounding of them."""
    obj, probe, loss = problem()
    want = torch.autograd.grad(loss(), (obj, probe))

    def close(got, factor=1.0):
        for a, b in zip(got, want):
            assert torch.linalg.norm(a - factor * b) <= 1e-6 * abs(factor) * torch.linalg.norm(b)

    value = loss()
    close(torch.autograd.grad(value, (obj, probe), retain_graph=True))
    close(torch.autograd.grad(2.0 * value, (obj, probe), retain_graph=True), 2.0)
    factor = torch.tensor(3.0, dtype=torch.float64, device="cuda", requires_grad=True)
    graph = torch.autograd.grad(value, (obj, probe), grad_outputs=factor, create_graph=True)
    close(graph, 3.0)
    (inner,) = torch.autograd.grad(torch.view_as_real(graph[0]).sum(), factor)
    assert abs(float(inner) - float(torch.view_as_real(want[0]).sum())) <= 1e-4 * float(want[0].abs().sum())
    batch = torch.autograd.grad(loss(), (obj, probe), grad_outputs=torch.tensor([1.0, -2.0], device="cuda").double(),
                                is_grads_batched=True)
    close([b[0] for b in batch])
    close([b[1] for b in batch], -2.0)
    with torch.autograd.graph.save_on_cpu():
        value = loss()
    close(torch.autograd.grad(value, (obj, probe)))
