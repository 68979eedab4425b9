"""Registration of spectra and images in the forms torch hands them out, and on two devices."""

from types import SimpleNamespace

import pytest
import torch


def spectra(count, h, w, seed=0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    base = torch.randn(h, w, generator=gen, device="cuda")
    shifted = [torch.roll(base, (3 * i, -2 * i), dims=(0, 1)) for i in range(count)]
    noise = 0.1 * torch.randn(count, h, w, generator=gen, device="cuda")
    return torch.fft.fft2(torch.stack(shifted) + noise)


@pytest.mark.gpu
@pytest.mark.parametrize("usfac", [0, 1, 2, 3, 100])
@pytest.mark.parametrize("sides", [(48, 40), (33, 51)])
@pytest.mark.parametrize("first, second", [(True, False), (False, True), (True, True)])
def test_conjugate_views(usfac, sides, first, second):
    """A lazily conjugated spectrum is the conjugate in memory: the same numbers, to the bit."""
    from ptychox_b200.registration import dftregistration

    s = spectra(5, *sides)
    a, b = s[0], s
    lazy = a.conj() if first else a, b.conj() if second else b
    assert lazy[0].is_conj() == first and lazy[1].is_conj() == second
    got = dftregistration(*lazy, usfac, return_registered=True)
    want = dftregistration(lazy[0].resolve_conj(), lazy[1].resolve_conj(), usfac, return_registered=True)
    for g, w in zip(got, want):
        assert torch.equal(g, w)


@pytest.mark.gpu
@pytest.mark.parametrize("view", ["negated", "imaginary"])
def test_negated_images(view):
    """A stack with the negative bit set, at a side of the library's own transforms and enough pixels
    for them: the positions of the same images in memory."""
    from ptychox_b200.registration import _prime_fft_bytes, track_position

    gen = torch.Generator(device="cuda").manual_seed(3)
    base = torch.rand(158, 158, generator=gen, device="cuda")
    images = torch.stack([torch.roll(base, (i % 7, -(i % 5)), dims=(0, 1)) for i in range(48)])
    assert _prime_fft_bytes(48, 118, 118) > 0
    if view == "negated":
        stack = torch._neg_view((-images).contiguous())
    else:
        stack = torch.imag(torch.complex(torch.zeros_like(images), -images).conj())
    assert stack.is_neg()
    for g, w in zip(track_position(stack, usfac=10, return_registered=True),
                    track_position(images, usfac=10, return_registered=True)):
        assert torch.equal(g, w)


def test_spectra_on_two_devices_are_refused():
    """Before anything is launched: the stand-ins hold nothing that a later step could use."""
    from ptychox_b200.registration import dftregistration

    a, b = (SimpleNamespace(ndim=2, is_cuda=True, shape=torch.Size((8, 8)), device=torch.device("cuda", i))
            for i in range(2))
    for usfac in (0, 1, 2, 100):
        with pytest.raises(ValueError, match="same device"):
            dftregistration(a, b, usfac)


@pytest.mark.gpu
@pytest.mark.parametrize("batch, rows, cols", [(1, 1, 1), (1, 255, 257), (1, 256, 256), (1, 1500, 1777), (3, 700, 701), (40, 181, 182),
                                               (700, 130, 129), (2, 1, 40000)])
def test_energies_of_few_and_many_images(batch, rows, cols):
    """One piece per image, several, and more than divide it evenly: within the rounding of an FP64 sum
    in any order, and the same on every call."""
    from ptychox_b200 import _abi
    from ptychox_b200.registration import _energy

    gen = torch.Generator(device="cuda").manual_seed(rows)
    spec = torch.randn(batch, rows, cols, dtype=torch.complex64, generator=gen, device="cuda")
    parts = _abi.query("ptx_reg_energy_parts", batch, rows, cols)
    assert 1 <= parts <= max(1, rows * cols // 2**15)
    want = torch.view_as_real(spec).double().square().sum(dim=(1, 2, 3))
    got = _energy(spec)
    eps = torch.finfo(torch.float64).eps
    assert ((got - want).abs() <= 4 * rows * cols * eps * want).all()
    assert torch.equal(got, _energy(spec))
