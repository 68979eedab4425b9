"""Line transforms of sides R p (p a prime of 37 to 127) against FP64 transforms: every R, the
smallest and largest p, line counts that end within a block, strided images, one image and a few;
and the rule that takes a stack there.

Tolerance: relative L2 below 1e-6 (plain FP32 sums of up to 64 pairs and up to 24-point
transforms: a few 1e-7)."""

import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu

SIDES = [(74, 111), (148, 185), (222, 296), (333, 370), (444, 74), (254, 381), (472, 118), (508, 82), (1016, 86), (122, 636)]


def lengths():
    from ptychox_b200 import _abi

    return lambda h, w: _abi.query("ptx_reg_prime_fft_workspace_bytes", h, w)


def spectra(images):
    from ptychox_b200._utils import call_on, ptr

    n, h, w = images.shape
    half, out = (torch.empty(n, *s, dtype=torch.complex64, device=images.device) for s in ((w, h), (h, w)))
    ws = torch.empty(lengths()(h, w), dtype=torch.uint8, device=images.device)
    call_on(images.device, "ptx_reg_prime_fft2", ptr(images), images.stride(0), images.stride(1), n, h, w, ptr(half),
            ptr(out), ptr(ws), ws.numel())
    return out.cpu().numpy()


@pytest.mark.parametrize("h, w", SIDES)
@pytest.mark.parametrize("count", [1, 3])
def test_spectra(h, w, count):
    rng = np.random.default_rng(h * 1000 + w)
    big = rng.random((count, h + 6, w + 5)).astype(np.float32)
    got = spectra(torch.from_numpy(big).cuda()[:, 3:3 + h, 2:2 + w])
    assert rel_l2(got, np.fft.fft2(big[:, 3:3 + h, 2:2 + w].astype(np.float64))) < 1e-6


@pytest.mark.parametrize("h, w", SIDES)
def test_correlation(h, w):
    from ptychox_b200._utils import call_on, ptr

    count = 2
    rng = np.random.default_rng(h * 1000 + w)
    q = (rng.standard_normal((count, h, w)) + 1j * rng.standard_normal((count, h, w))).astype(np.complex64)
    padded = np.zeros((count, 2 * h, 2 * w), np.complex128)
    r0, c0 = h - h // 2, w - w // 2
    padded[:, r0:r0 + h, c0:c0 + w] = np.fft.fftshift(q.conj(), axes=(1, 2))
    want = np.fft.ifft2(np.fft.ifftshift(padded, axes=(1, 2)), norm="forward").transpose(0, 2, 1)
    dev = torch.device("cuda", torch.cuda.current_device())
    x = torch.from_numpy(q).cuda()
    half, out = (torch.empty(count, 2 * w, n, dtype=torch.complex64, device=dev) for n in (h, 2 * h))
    ws = torch.empty(lengths()(h, w), dtype=torch.uint8, device=dev)
    call_on(dev, "ptx_reg_prime_correlation", ptr(x), count, h, w, ptr(half), ptr(out), ptr(ws), ws.numel())
    assert rel_l2(out.cpu().numpy(), want) < 1e-6
    with pytest.raises(Exception, match="workspace"):
        call_on(dev, "ptx_reg_prime_correlation", ptr(x), count, h, w, ptr(half), ptr(out), ptr(ws), ws.numel() - 1)
    assert lengths()(h, 480) == 0


@pytest.mark.parametrize("n, h, w", [(4, 480, 480), (9, 259, 259), (200, 113, 74), (3, 481, 481), (2, 472, 472)])
def test_other_stacks_stay_on_the_library(n, h, w):
    from ptychox_b200 import registration

    assert registration._prime_fft_bytes(n, h, w) == 0
    x = torch.rand(n, h, w, device="cuda")
    assert torch.equal(registration._spectra(x), torch.fft.fft2(x.to(torch.complex64)))


def test_positions_layouts_and_gradients():
    """Tracking at a side of 8 x 41 equals the library transforms' positions, also for a stack with
    another order of the axes; one that requires grad keeps its graph, one under vmap or forward-mode
    differentiation its derivatives."""
    from torch.autograd import forward_ad

    from ptychox_b200 import registration

    g = torch.Generator(device="cuda").manual_seed(5)
    base = torch.rand(400, 400, device="cuda", generator=g)
    base = torch.nn.functional.avg_pool2d(base[None, None], 5, 1, 2)[0, 0]
    stack = torch.stack([torch.roll(base, (i, -2 * i), (0, 1))[:368, :368] for i in range(5)])
    assert registration._prime_fft_bytes(5, 328, 328) > 0
    x, y = registration.track_position(stack)
    crop = stack[:, 20:-20, 20:-20]
    ref_spectra = torch.fft.fft2(crop.to(torch.complex64))
    ref = registration.dftregistration(ref_spectra[:1], ref_spectra[:1].expand(2, -1, -1), 600)  # below the rule's size
    assert float(x[0]) == float(ref[0, 3]) and float(y[0]) == float(ref[0, 2])
    want = torch.fft.fft2(crop.double()).cpu().numpy()
    assert rel_l2(registration._spectra(crop).cpu().numpy(), want) < 1e-6
    across = registration._spectra(crop.transpose(1, 2))
    assert rel_l2(across.cpu().numpy(), want.transpose(0, 2, 1)) < 1e-6
    assert float((x.abs() - 2 * torch.arange(5, device="cuda")).abs().max()) < 0.02
    leaf = stack.clone().requires_grad_(True)
    registration.track_position(leaf, return_registered=True)[2].abs().sum().backward()
    assert leaf.grad is not None
    with forward_ad.dual_level():
        dual = forward_ad.make_dual(crop, torch.ones_like(crop))
        assert forward_ad.unpack_dual(registration._spectra(dual)).tangent is not None
    twice = torch.vmap(registration._spectra)(torch.stack([crop, crop]))
    assert rel_l2(twice[1].cpu().numpy(), want) < 1e-6
