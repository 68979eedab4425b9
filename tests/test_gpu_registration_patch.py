"""The upsampled correlation patch and its peak (``ptx_reg_upsampled_peak``) against the dense
FP64 transform, at the edges of its tiles: one-line spectra, 32-column and 64-row stages, patches
one point around a 64-point tile, a single and a shared row block; and the passes of the initial
estimate against numpy.

Tolerance: both sides sum ``rows * cols`` FP64 terms of total magnitude ``S = sum |Q|`` in some
order, each term a product of a few rounded factors, so each is within ``32 eps S`` of the exact
value (pairwise or random-walk growth is far smaller); the two differ by at most ``64 eps S``, and the point
found is a maximum of the dense patch up to twice that.
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def phases(length, points):
    """Centred frequency times point, ``[length, points]``."""
    k = np.arange(length)
    return np.where(k < (length + 1) // 2, k, k - length)[:, None] * points[None, :]


@pytest.mark.parametrize("rows, cols, usfac", [(1, 1, 3), (1, 33, 5), (64, 32, 4), (65, 31, 42), (63, 97, 43),
                                               (45, 50, 9), (130, 64, 85), (40, 72, 600)])
@pytest.mark.parametrize("batch", [1, 5])
def test_patch_peak_is_the_dense_transforms(rows, cols, usfac, batch):
    from ptychox_b200 import _abi
    from ptychox_b200._utils import ptr, stream_handle, workspace

    rng = np.random.default_rng(1000 * rows + cols + usfac)
    q = (rng.standard_normal((batch, rows, cols)) + 1j * rng.standard_normal((batch, rows, cols))).astype(np.complex64)
    centre = rng.integers(-3 * usfac, 3 * usfac + 1, size=(2, batch)).astype(np.int32)
    dev = torch.device("cuda:0")
    tq, trc, tcc = (torch.from_numpy(a).to(dev) for a in (q, centre[0], centre[1]))
    peak = torch.empty(batch, 2, dtype=torch.int32, device=dev)
    value = torch.empty(batch, dtype=torch.complex128, device=dev)
    ws = workspace(_abi.query("ptx_reg_workspace_bytes", batch, rows, cols, usfac), dev)
    _abi.call("ptx_reg_upsampled_peak", ptr(tq), batch, rows, cols, usfac, ptr(trc), ptr(tcc), ptr(peak), ptr(value),
              ptr(ws), ws.numel(), stream_handle(dev))
    n = (3 * usfac + 1) // 2
    at = np.arange(n) - n // 2
    for b in range(batch):
        kr, kc = (np.exp(-2j * np.pi * (phases(length, at + c) % (length * usfac)) / (length * usfac))
                  for length, c in ((rows, int(centre[0, b])), (cols, int(centre[1, b]))))
        cc = np.conj(kr.T @ q[b].astype(np.complex128) @ kc)
        tol = 64 * np.finfo(np.float64).eps * np.abs(q[b].astype(np.complex128)).sum()
        r, c = peak[b].cpu().numpy()
        assert abs(complex(value[b].cpu()) - cc[r, c]) <= tol
        assert abs(cc[r, c]) >= np.abs(cc).max() - 2 * tol


def test_ties_take_the_first_point_and_nan_the_origin():
    """A constant image's patch is constant (every tie: the first point in column-major order);
    a spectrum with a NaN has no maximum (the first point, value NaN)."""
    from ptychox_b200 import _abi
    from ptychox_b200._utils import ptr, stream_handle, workspace

    dev = torch.device("cuda:0")
    q = torch.zeros(2, 48, 40, dtype=torch.complex64, device=dev)
    q[:, 0, 0] = 3.0
    q[1, 5, 7] = float("nan")
    zero = torch.zeros(2, dtype=torch.int32, device=dev)
    peak = torch.full((2, 2), -1, dtype=torch.int32, device=dev)
    value = torch.zeros(2, dtype=torch.complex128, device=dev)
    ws = workspace(_abi.query("ptx_reg_workspace_bytes", 2, 48, 40, 100), dev)
    _abi.call("ptx_reg_upsampled_peak", ptr(q), 2, 48, 40, 100, ptr(zero), ptr(zero), ptr(peak), ptr(value), ptr(ws),
              ws.numel(), stream_handle(dev))
    assert peak.cpu().tolist() == [[0, 0], [0, 0]]
    assert complex(value[0].cpu()) == 3.0 and np.isnan(complex(value[1].cpu()).real)


@pytest.mark.parametrize("rows, cols", [(1, 1), (1, 40), (33, 1), (16, 31), (48, 64), (45, 51), (97, 130)])
@pytest.mark.parametrize("single", [True, False])
def test_half_pixel_estimate(rows, cols, single):
    """Peak of the twice-upsampled correlation, cross-power and energies.  The correlation is an
    FP32 transform of ``rows * cols`` products: its values are within ``32 eps32 sum |product|``
    of the FP64 transform's (a few rounded stages per axis), so the peak is a maximum of it up
    to twice that."""
    from ptychox_b200.registration import _energy, _half_pixel_estimate

    rng = np.random.default_rng(rows * 1000 + cols)
    b, usfac = 3, 7
    s1 = rng.standard_normal((1 if single else b, rows, cols, 2)).astype(np.float32).view(np.complex64)[..., 0]
    s2 = rng.standard_normal((b, rows, cols, 2)).astype(np.float32).view(np.complex64)[..., 0]
    t1, t2 = torch.from_numpy(s1).cuda(), torch.from_numpy(s2).cuda()
    half, centre, value, q = (t.cpu().numpy() for t in _half_pixel_estimate(t1, t2, usfac))
    product = s1.astype(np.complex128) * np.conj(s2.astype(np.complex128))
    assert np.abs(q - np.conj(product)).max() <= 4 * np.finfo(np.float32).eps * np.abs(product).max()
    full = np.zeros((b, 2 * rows, 2 * cols), np.complex128)
    full[:, rows - rows // 2:2 * rows - rows // 2, cols - cols // 2:2 * cols - cols // 2] = np.fft.fftshift(
        product, axes=(1, 2))
    corr = np.fft.ifft2(np.fft.ifftshift(full, axes=(1, 2))) * (4 * rows * cols)
    for i in range(b):
        r, c = half[i]
        assert -rows <= r < rows and -cols <= c < cols
        tol = 32 * np.finfo(np.float32).eps * np.abs(product[i]).sum()
        assert abs(value[i] - corr[i, r, c]) <= tol
        assert abs(corr[i, r, c]) >= np.abs(corr[i]).max() - 2 * tol
        want = [np.sign(v) * np.floor(abs(v) * usfac / 2 + 0.5) for v in (r, c)]
        assert centre[:, i].tolist() == want
    energy = _energy(t2).cpu().numpy()
    exact = (np.abs(s2.astype(np.complex128)) ** 2).sum(axis=(1, 2))
    assert np.abs(energy - exact).max() <= 4 * rows * cols * np.finfo(np.float64).eps * exact.max()
