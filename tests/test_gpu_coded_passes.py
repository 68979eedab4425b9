"""The persistent coded passes at the edges of their work splits and rules, against the FP64
oracle: one frame and a few (fewer units than CTAs), as many frames as the shift-ramp tables
hold and one more (the passes then evaluate the ramp), every downsampling factor, transfer
functions off a 16-byte boundary, and gradients computed in place of the object.

Tolerance: relative L2 below 1e-5, or five times the error of the oracle's complex64 formulation
where that misses it (the ramps and transforms round differently in the two)."""

import numpy as np
import pytest
import torch

from conftest import rel_l2
from oracle import ptycho_oracle as O

pytestmark = pytest.mark.gpu


def cuda(a, offset=0):
    """The array on the GPU, `offset` elements past an aligned address."""
    if a is None:
        return None
    t = torch.from_numpy(np.ascontiguousarray(a))
    room = torch.empty(t.numel() + offset, dtype=t.dtype, device="cuda")
    out = room[offset:].view(t.shape)
    out.copy_(t)
    return out


def problem(n, count, ds, nearfield):
    from ptychox_b200 import synth

    rng = np.random.default_rng(n * 100 + count)
    obj, mask = synth.random_object(n, n, rng), synth.binary_mask(n, 0.5, rng)
    t2 = synth.angular_spectrum_transfer(n, 1.85e-6, 0.5e-6, 2e-3)
    t1 = None if nearfield else synth.angular_spectrum_transfer(n, 1.85e-6, 0.5e-6, 396.95e-6)
    shifts = synth.coded_shifts(count, 5.0, n, rng)
    amp = O.coded_forward(obj, mask, t1, t2, shifts, ds)[3]
    meas, scale = synth.poisson_counts(amp**2, 1e3, rng, per_pixel=True)
    guess = (0.8 * obj * (1 + 0.3 * rng.standard_normal(obj.shape))).astype(np.complex64)
    return guess, mask, t1, t2, shifts.astype(np.float32), meas, scale


def check(got, args, ds, loss="mse"):
    guess, mask, t1, t2, shifts, meas, scale = args
    want = O.coded_sweep(guess, mask, t1, t2, shifts, ds, meas, scale, loss=loss, with_shifts=True)
    ref32 = O.coded_sweep(guess, mask, t1, t2, shifts, ds, meas, scale, fp64=False, loss=loss, with_shifts=True)
    assert abs(float(got[0]) - want[0]) <= 1e-5 * abs(want[0])
    for g, w, r in zip(got[1:], want[1:], ref32[1:]):
        assert rel_l2(g.cpu().numpy(), w) < max(1e-5, 5 * rel_l2(r, w))


@pytest.mark.parametrize("n, count", [(16, 1), (16, 8), (16, 9), (32, 17), (64, 3), (256, 2), (1024, 1), (60, 30), (60, 31)])
@pytest.mark.parametrize("nearfield", [False, True])
def test_sweep(n, count, nearfield):
    from ptychox_b200.coded import coded_sweep

    args = problem(n, count, 2, nearfield)
    guess, mask, t1, t2, shifts, meas, scale = args
    got = coded_sweep(cuda(guess), cuda(mask), cuda(t1), cuda(t2), cuda(shifts), 2, cuda(meas), scale, with_shifts=True)
    check(got, args, 2)


@pytest.mark.parametrize("ds", [1, 2, 4, 8])
@pytest.mark.parametrize("loss", ["mse", "fd-isotropic"])
def test_downsampling_and_unaligned_transfer(ds, loss):
    from ptychox_b200.coded import coded_sweep

    args = problem(128, 5, ds, False)
    guess, mask, t1, t2, shifts, meas, scale = args
    got = coded_sweep(cuda(guess), cuda(mask), cuda(t1, 1), cuda(t2, 1), cuda(shifts), ds, cuda(meas), scale, loss=loss,
                      with_shifts=True)
    check(got, args, ds, loss)


def test_gradient_in_place_of_the_object():
    from ptychox_b200 import _abi
    from ptychox_b200._utils import call_on, ptr, workspace

    args = problem(64, 4, 2, False)
    guess, mask, t1, t2, shifts, meas, scale = args
    dev = torch.device("cuda", torch.cuda.current_device())
    obj, m, a, b, sh, y = (cuda(x) for x in (guess, mask, t1, t2, shifts, meas))
    loss, gm = torch.empty((), dtype=torch.float64, device=dev), torch.empty_like(m)
    ws = workspace(_abi.query("ptx_coded_workspace_bytes", 64, 4), dev)
    call_on(dev, "ptx_coded_sweep", ptr(obj), ptr(m), ptr(a), ptr(b), 64, ptr(sh), 4, 2, ptr(y), scale, ptr(loss),
            ptr(obj), ptr(gm), ptr(ws), ws.numel())
    check((loss, obj, gm), args, 2)


@pytest.mark.parametrize("n, ds, count", [
    (18, 3, 9),     # fewer columns than three strips, the last one partial
    (25, 5, 12),    # odd: rows off 16 bytes, as many frames as the ramp tables hold
    (25, 1, 13),    # and one more
    (27, 27, 3),    # one pooled row
    (45, 3, 2),
    (75, 15, 4),    # row groups that end past the last row
    (100, 2, 5),
    (243, 9, 2),
    (625, 1, 1),    # 25 x 25
    (972, 6, 1),
    (1000, 8, 2),
])
@pytest.mark.parametrize("nearfield", [False, True])
def test_mixed_radix_edges(n, ds, count, nearfield):
    from ptychox_b200.coded import coded_sweep

    args = problem(n, count, ds, nearfield)
    guess, mask, t1, t2, shifts, meas, scale = args
    got = coded_sweep(cuda(guess), cuda(mask), cuda(t1, 1), cuda(t2, 1), cuda(shifts), ds, cuda(meas), scale,
                      with_shifts=True)
    check(got, args, ds)


@pytest.mark.parametrize("n, ds", [(60, 4), (45, 3)])
def test_mixed_radix_backward_of_unaligned_buffers(n, ds):
    """The adjoint on a sensor field that starts 8 bytes off a 16-byte boundary; x there is refused."""
    from ptychox_b200 import _abi
    from ptychox_b200._utils import call_on, ptr, workspace

    count = 3
    guess, mask, t1, t2, shifts, _, _ = problem(n, count, ds, False)
    _, xf, sensor, amp = O.coded_forward(guess, mask, t1, t2, shifts, ds)
    gout = np.random.default_rng(n).standard_normal(amp.shape).astype(np.float32)
    want = O.coded_backward(gout, xf, sensor, amp, mask, t1, t2, shifts, ds)
    dev = torch.device("cuda", torch.cuda.current_device())
    g, a, m, x1, x2, sh = (cuda(v) for v in (gout, amp.astype(np.float32), mask, t1, t2, shifts))
    off, xc, sc = (cuda(v.astype(np.complex64), o) for v, o in ((xf, 1), (xf, 0), (sensor, 1)))
    go, gm = torch.empty_like(m), torch.empty_like(m)
    ws = workspace(_abi.query("ptx_coded_workspace_bytes", n, count), dev)

    def backward(x):
        call_on(dev, "ptx_coded_backward", ptr(g), ptr(x), ptr(sc), ptr(a), ptr(m), ptr(x1), ptr(x2), n, ptr(sh), count,
                ds, ptr(go), ptr(gm), ptr(ws), ws.numel())

    with pytest.raises(ValueError):
        backward(off)
    backward(xc)
    for got, ref in zip((go, gm), want):
        assert rel_l2(got.cpu().numpy(), ref) < 1e-5
