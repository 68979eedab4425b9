"""Sub-pixel image registration for positional tracking of coded / near-field scans.

Mirrors the MATLAB helpers of the reference's near-field example
(``matlab/Examples/Near-field Ptychography/+misc``):

* ``dftregistration`` — ``dftregistration.m:70-138``: efficient sub-pixel registration by
  cross-correlation (M. Guizar-Sicairos, S. T. Thurman and J. R. Fienup, Opt. Lett. 33,
  156-158 (2008)), batched over images;
* ``track_position`` — ``track_position.m:24-41`` (register every measurement against
  the first, 20-pixel border removed, ``usfac = 600``);
* ``refine_position`` — ``refine_position.m:25-55`` (register against the average of the
  measurements shifted back by their initial estimates, ``usfac = 100``).

Stacks are ``[n, h, w]`` (the MATLAB functions take ``[h, w, n]``); shifts are
``(row, col)`` as in the reference, and the trackers return ``(locX, locY)`` =
``(col, row)``.  The plain FFTs of images and of the 2x zero-padded cross-correlation run in
libptychox where a side has a prime factor that cuFFT is slow at (``ptx_reg_prime_*``), else on
cuFFT (``torch.fft``); the passes around them, the matrix-multiply DFT refinement (``dftups``,
``:150-185``, summed in FP64) and both peak searches run in libptychox (``ptx_reg_*``).
FP32 spectra and FFTs, FP64 energy sums.
"""

from __future__ import annotations

import math

import torch

from . import _abi
from ._utils import ptr, readable, stream_handle, workspace

__all__ = ["dftregistration", "track_position", "refine_position"]

# Pixels of a stack from which the library's prime-factor transforms are taken: one 472 x 472 image
# takes 33 us there against 28 on cuFFT (four launches), 64 of 118 x 118 41 against 58.
_PRIME_FFT_PIXELS = 1 << 19
_WS_CAP = 2 << 30  # refinement workspace per library call; larger batches are split


def _freq(n: int, device) -> torch.Tensor:
    """``ifftshift(-fix(n/2):ceil(n/2)-1)`` (``dftregistration.m:73-74``)."""
    return torch.fft.ifftshift(torch.arange(-(n // 2), (n + 1) // 2, device=device))


def _argmax_colmajor(a: torch.Tensor) -> tuple[torch.Tensor, torch.Tensor]:
    """(row, col) of the first maximum of each ``[B, R, C]`` slice in column-major order
    (MATLAB's ``find(A == max(A(:)), 1, 'first')``)."""
    rows = a.shape[1]
    idx = a.transpose(1, 2).reshape(a.shape[0], -1).argmax(dim=1)
    return idx % rows, idx // rows


def _ftpad2(spec: torch.Tensor) -> torch.Tensor:
    """``FTpad(spec, [2 nr, 2 nc])`` (``dftregistration.m:189-224``) for ``[B, nr, nc]``."""
    b, nr, nc = spec.shape
    out = torch.zeros(b, 2 * nr, 2 * nc, dtype=spec.dtype, device=spec.device)
    r0, c0 = nr - nr // 2, nc - nc // 2
    out[:, r0:r0 + nr, c0:c0 + nc] = torch.fft.fftshift(spec, dim=(-2, -1))
    return torch.fft.ifftshift(out, dim=(-2, -1)) * 4.0


def _prime_fft_bytes(count: int, h: int, w: int) -> int:
    """Workspace of the library's prime-factor transforms, 0 where cuFFT is to be taken."""
    return _abi.query("ptx_reg_prime_fft_workspace_bytes", h, w) if count * h * w >= _PRIME_FFT_PIXELS else 0


def _half_pixel_estimate(b1: torch.Tensor, b2: torch.Tensor, usfac: int):
    """Peak of the cross-correlation of ``b1`` (one image or as many as ``b2``) and ``b2``
    upsampled twice (``dftregistration.m:90-101``, ``FTpad`` ``:189-224``): signed half pixels
    ``[B, 2]``, the centres ``round(shift usfac)``, the unnormalised correlation there, and the
    cross-power spectrum.  The inverse transform is taken line by line, along the rows before
    they are padded and along the columns after."""
    bsz, nr, nc = b2.shape
    dev = b2.device
    stream = stream_handle(dev)
    with torch.cuda.device(dev):
        q = torch.empty(bsz, nr, nc, dtype=torch.complex64, device=dev)
        corr = torch.empty(bsz, 2 * nc, 2 * nr, dtype=torch.complex64, device=dev)
        own = _prime_fft_bytes(bsz, nr, nc)
        if own:
            _abi.call("ptx_reg_cross_power", ptr(b1), b1.shape[0], ptr(b2), bsz, nr, nc, None, ptr(q), stream)
            rows = torch.empty(bsz, 2 * nc, nr, dtype=torch.complex64, device=dev)
            tables = torch.empty(own, dtype=torch.uint8, device=dev)
            _abi.call("ptx_reg_prime_correlation", ptr(q), bsz, nr, nc, ptr(rows), ptr(corr), ptr(tables), own, stream)
        else:
            rows = torch.empty(bsz, nr, 2 * nc, dtype=torch.complex64, device=dev)
            _abi.call("ptx_reg_cross_power", ptr(b1), b1.shape[0], ptr(b2), bsz, nr, nc, ptr(rows), ptr(q), stream)
            rows = torch.fft.ifft(rows, norm="forward")
            _abi.call("ptx_reg_pad_transpose", ptr(rows), bsz, nr, nc, ptr(corr), stream)
            corr = torch.fft.ifft(corr, norm="forward")
        half = torch.empty(bsz, 2, dtype=torch.int32, device=dev)
        centre = torch.empty(2, bsz, dtype=torch.int32, device=dev)
        value = torch.empty(bsz, dtype=torch.complex128, device=dev)
        ws = workspace(_abi.query("ptx_reg_estimate_workspace_bytes", bsz, nr, nc), dev)
        _abi.call("ptx_reg_estimate", ptr(corr), bsz, nr, nc, usfac, ptr(half), ptr(centre[0]), ptr(centre[1]),
                  ptr(value), ptr(ws), ws.numel(), stream)
    return half, centre, value, q


def _in_memory(t: torch.Tensor) -> torch.Tensor:
    """``t`` contiguous with a lazy conjugation or negation carried out: a pointer sees neither."""
    return t.contiguous().resolve_conj().resolve_neg()


def _plain(t: torch.Tensor) -> bool:
    """Whether the library may read ``t`` directly, and no derivative is wanted of it."""
    return readable(t) and not (t.requires_grad and torch.is_grad_enabled())


def _energy(spec: torch.Tensor) -> torch.Tensor:
    """``sum |spec|^2`` of each image in FP64."""
    if spec.numel() and not _plain(spec):
        return (spec.abs().double() ** 2).sum(dim=(-2, -1))
    with torch.cuda.device(spec.device):
        parts = _abi.query("ptx_reg_energy_parts", *spec.shape)
        out = torch.empty(spec.shape[0], parts, dtype=torch.float64, device=spec.device)
        _abi.call("ptx_reg_partial_energy", ptr(spec), *spec.shape, parts, ptr(out), stream_handle(spec.device))
    return out.sum(dim=1) if parts > 1 else out[:, 0]


def _refine(q: torch.Tensor, usfac: int, rc: torch.Tensor, cc: torch.Tensor):
    """Peak (row, col) of the upsampled patch and CC there, through the library."""
    b, nr, nc = q.shape
    peak_rc = torch.empty(b, 2, dtype=torch.int32, device=q.device)
    peak_cc = torch.empty(b, dtype=torch.complex128, device=q.device)
    per_image = max(1, _abi.query("ptx_reg_workspace_bytes", 1, nr, nc, usfac))
    step = max(1, min(b, _WS_CAP // per_image))
    ws = workspace(per_image * step, q.device)
    with torch.cuda.device(q.device):
        for s in range(0, b, step):
            e = min(b, s + step)
            _abi.call("ptx_reg_upsampled_peak", ptr(q[s:e]), e - s, nr, nc, int(usfac), ptr(rc[s:e]), ptr(cc[s:e]),
                      ptr(peak_rc[s:e]), ptr(peak_cc[s:e]), ptr(ws), ws.numel(), stream_handle(q.device))
    return peak_rc.long(), peak_cc


def dftregistration(buf1ft: torch.Tensor, buf2ft: torch.Tensor, usfac: int = 1, return_registered: bool = False):
    """``[error, diffphase, row_shift, col_shift]`` registering ``buf2ft`` to ``buf1ft``.

    ``buf1ft`` / ``buf2ft``: complex spectra (``fft2`` of the images) on the GPU, ``[h, w]``
    or ``[B, h, w]`` (a single spectrum on either side is broadcast).  ``usfac``: 0 (error
    and phase only), 1 (whole pixels), 2 (half pixels) or larger (1/usfac of a pixel).
    Returns float64 ``[B, 4]``, or ``[4]`` when both inputs are 2-D; with
    ``return_registered`` also ``Greg``, the spectrum of ``buf2ft`` shifted and phase-corrected
    onto ``buf1ft`` (the second output of ``dftregistration.m:140-148``), complex64.
    """
    if buf1ft.ndim not in (2, 3) or buf2ft.ndim not in (2, 3):
        raise ValueError("buf1ft and buf2ft must be [h, w] or [batch, h, w] spectra.")
    if not buf1ft.is_cuda or not buf2ft.is_cuda:
        raise ValueError("buf1ft and buf2ft must be CUDA tensors (ptychox_b200 has no CPU path).")
    if buf1ft.shape[-2:] != buf2ft.shape[-2:]:
        raise ValueError("buf1ft and buf2ft must have the same image size.")
    if buf1ft.device != buf2ft.device:
        raise ValueError("buf1ft and buf2ft must live on the same device.")
    usfac = int(usfac)
    if usfac < 0:
        raise ValueError("usfac must be non-negative.")
    single = buf1ft.ndim == 2 and buf2ft.ndim == 2
    b1 = buf1ft.to(torch.complex64).reshape(-1, *buf1ft.shape[-2:])
    b2 = buf2ft.to(torch.complex64).reshape(-1, *buf2ft.shape[-2:])
    bsz = max(b1.shape[0], b2.shape[0])
    b1, b2 = _in_memory(b1.expand(min(bsz, b1.shape[0]), -1, -1)), _in_memory(b2.expand(bsz, -1, -1))
    if b1.shape[0] not in (1, bsz):
        b1 = b1.expand(bsz, -1, -1)  # raises: the two batches differ
    nr, nc = b2.shape[-2:]
    dev = b2.device
    zeros = torch.zeros(bsz, dtype=torch.float64, device=dev)
    if usfac == 0:
        ccmax = (b1.to(torch.complex128) * b2.to(torch.complex128).conj()).sum(dim=(-2, -1))
        row_shift, col_shift = zeros, zeros.clone()
    elif usfac == 1:
        cc = torch.fft.ifft2(b1 * b2.conj())
        r, c = _argmax_colmajor(cc.abs())
        ccmax = cc[torch.arange(bsz, device=dev), r, c].to(torch.complex128) * (nr * nc)
        row_shift, col_shift = _freq(nr, dev)[r].double(), _freq(nc, dev)[c].double()
    elif usfac == 2 and b2.numel() and not (_plain(b1) and _plain(b2)):
        cc = torch.fft.ifft2(_ftpad2(b1 * b2.conj()))
        r, c = _argmax_colmajor(cc.abs())
        ccmax = cc[torch.arange(bsz, device=dev), r, c].to(torch.complex128) * (nr * nc)
        row_shift, col_shift = (torch.fft.ifftshift(torch.arange(-n, n, device=dev))[i].double() / 2.0
                                for n, i in ((nr, r), (nc, c)))
    else:
        half, centre, ccmax, q = _half_pixel_estimate(b1.detach(), b2.detach(), usfac)
        row_shift, col_shift = half[:, 0].double() / 2.0, half[:, 1].double() / 2.0
        if usfac > 2:
            peak, ccmax = _refine(q, usfac, centre[0], centre[1])
            dftshift = math.ceil(1.5 * usfac) // 2
            row_shift = centre[0].double() / usfac + (peak[:, 0] - dftshift).double() / usfac
            col_shift = centre[1].double() / usfac + (peak[:, 1] - dftshift).double() / usfac
    if usfac > 1:
        if nr == 1:
            row_shift = zeros
        if nc == 1:
            col_shift = zeros.clone()
    error = torch.sqrt(torch.abs(1.0 - ccmax.abs() ** 2 / (_energy(b1) * _energy(b2))))
    diffphase = torch.angle(ccmax)
    out = torch.stack([error, diffphase, row_shift, col_shift], dim=1)
    if not return_registered:
        return out[0] if single else out
    fr = _freq(nr, dev).double()[None, :, None] / nr
    fc = _freq(nc, dev).double()[None, None, :] / nc
    phase = diffphase[:, None, None]
    if usfac > 0:
        phase = phase - 2 * math.pi * (row_shift[:, None, None] * fr + col_shift[:, None, None] * fc)
    greg = b2 * torch.polar(torch.ones_like(phase), phase).to(torch.complex64)
    return (out[0], greg[0]) if single else (out, greg)


def _crop(stack: torch.Tensor, edge: int) -> torch.Tensor:
    return stack[..., edge:stack.shape[-2] - edge, edge:stack.shape[-1] - edge]


def _spectra(images: torch.Tensor) -> torch.Tensor:
    """``fft2`` of real images ``[..., h, w]``, complex64."""
    h, w = images.shape[-2:]
    own = _prime_fft_bytes(images.numel() // max(1, h * w), h, w)
    if own:
        images = images.resolve_neg()
    if not own or images.dtype != torch.float32 or not _plain(images):
        return torch.fft.fft2(images.to(torch.complex64))
    x = images.reshape(-1, h, w)
    if x.stride(2) != 1:
        x = x.contiguous()
    half = torch.empty(x.shape[0], w, h, dtype=torch.complex64, device=x.device)
    out = torch.empty(*images.shape, dtype=torch.complex64, device=x.device)
    tables = torch.empty(own, dtype=torch.uint8, device=x.device)
    with torch.cuda.device(x.device):
        _abi.call("ptx_reg_prime_fft2", ptr(x), x.stride(0), x.stride(1), x.shape[0], h, w, ptr(half), ptr(out),
                  ptr(tables), own, stream_handle(x.device))
    return out


def _check_stack(im_raw_crop: torch.Tensor, edge: int) -> torch.Tensor:
    if im_raw_crop.ndim != 3:
        raise ValueError("im_raw_crop must be an [n, h, w] stack.")
    if not im_raw_crop.is_cuda:
        raise ValueError("im_raw_crop must be a CUDA tensor (ptychox_b200 has no CPU path).")
    if min(im_raw_crop.shape[-2:]) <= 2 * edge:
        raise ValueError(f"images must be larger than twice the {edge}-pixel border.")
    return im_raw_crop.to(torch.float32)


def track_position(im_raw_crop: torch.Tensor, edge: int = 20, usfac: int = 600, return_registered: bool = False):
    """Initial positional tracking (``track_position.m:24-41``): every measurement of the
    ``[n, h, w]`` stack registered against the first, ``edge`` pixels of border removed.
    Returns float64 ``(locX, locY)``, and with ``return_registered`` also ``regi``, the
    registered spectra of the cropped measurements (``[n, h - 2 edge, w - 2 edge]``)."""
    stack = _check_stack(im_raw_crop, edge)
    spectra = _spectra(_crop(stack, edge))
    res = dftregistration(spectra[0], spectra, usfac, return_registered=return_registered)
    if return_registered:
        out, regi = res
        return out[:, 3], out[:, 2], regi
    return res[:, 3], res[:, 2]


def refine_position(im_raw_crop: torch.Tensor, loc_x0, loc_y0, edge: int = 20, usfac: int = 100):
    """Positional refinement (``refine_position.m:25-55``): the stack is normalised by its
    mean image; the measurements whose initial shifts both exceed 2 pixels in magnitude are
    shifted back by them (Fourier phase ramp) and averaged (magnitude) into a reference, and
    every measurement is registered against it.  Returns float64 ``(locX, locY)``."""
    stack = _check_stack(im_raw_crop, edge)
    stack = stack / stack.mean(dim=0, keepdim=True)
    n, h, w = stack.shape
    dev = stack.device
    x0 = torch.as_tensor(loc_x0, dtype=torch.float64, device=dev).reshape(n)
    y0 = torch.as_tensor(loc_y0, dtype=torch.float64, device=dev).reshape(n)
    fy = _freq(h, dev).double()[:, None]
    fx = _freq(w, dev).double()[None, :]
    use = torch.nonzero((x0.abs() > 2) & (y0.abs() > 2)).flatten()
    ref = torch.zeros(h, w, dtype=torch.complex64, device=dev)
    for s in range(0, use.numel(), 64):
        idx = use[s:s + 64]
        hs = torch.exp(-2j * math.pi * (fx * x0[idx, None, None] / w + fy * y0[idx, None, None] / h))
        ref += torch.fft.ifft2(torch.fft.fft2(stack[idx].to(torch.complex64)) * hs.to(torch.complex64)).sum(dim=0)
    ref_img = ref.abs() / n
    ref_ft = _spectra(_crop(ref_img, edge))
    out = dftregistration(ref_ft, _spectra(_crop(stack, edge)), usfac)
    return out[:, 3], out[:, 2]
