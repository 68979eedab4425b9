"""The 512-point column pipeline and the persistent sub-pixel row passes at the edges of their
work splits, against the FP64 oracle: fewer tiles than CTAs, one tile more than a wave, a
frame one tile pair wide, counts off a 16-byte boundary (the unpipelined pass), row counts that
the row groups do not divide, one and several frames.  Tolerance: relative L2 below 1e-5, as in
the other oracle tests (the reference's FP32 formulation is an order below it at these sizes)."""

import numpy as np
import pytest
import torch

from conftest import rel_l2
from oracle import ptycho_oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-5


def cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def problem(ph, pw, count, seed, subpixel=False):
    from ptychox_b200 import synth

    rng = np.random.default_rng(seed)
    h, w = ph + 40, pw + 50
    obj, probe = synth.random_object(h, w, rng), synth.gaussian_probe(ph, pw, rng)
    pos = np.stack([rng.uniform(0, w - pw - 0.51, count), rng.uniform(0, h - ph - 0.51, count)], axis=1)
    if not subpixel:
        pos = pos.astype(np.int64)
    amp = (O.base_subpix_forward if subpixel else O.base_forward)(obj, probe, pos, fp64=False)[0]
    meas, scale = synth.poisson_counts(amp.astype(np.float64) ** 2, 2.0 * ph * pw, rng)
    guess = (0.9 * obj * (1 + 0.2 * rng.standard_normal(obj.shape))).astype(np.complex64)
    return guess, probe, pos, meas, scale


def check(got, want):
    loss, g1, g2 = (t.cpu().numpy() for t in got)
    assert abs(float(loss) - want[0]) <= TOL * abs(want[0])
    assert rel_l2(g1, want[1]) < TOL and rel_l2(g2, want[2]) < TOL


@pytest.mark.parametrize("pw, count", [(32, 1), (32, 74), (32, 75), (64, 3), (512, 2), (96, 5)])
@pytest.mark.parametrize("offset", [0, 1])
def test_column_pipeline(pw, count, offset):
    from ptychox_b200.base import base_sweep

    guess, probe, pos, meas, scale = problem(512, pw, count, 7 * pw + count)
    room = torch.empty(meas.size + offset, dtype=torch.uint16, device="cuda")
    counts = room[offset:].view(meas.shape)
    counts.copy_(cuda(meas))
    check(base_sweep(cuda(guess), cuda(probe), cuda(pos), counts, scale), O.base_sweep(guess, probe, pos, meas, scale))


def test_column_pipeline_of_the_fourier_sweep():
    from ptychox_b200 import synth
    from ptychox_b200.fpm import fpm_sweep

    rng = np.random.default_rng(3)
    obj, pupil = synth.random_object(1024, 1024, rng), synth.circular_pupil(512, 0.3)
    led = np.array([[256, 256], [200, 310], [300, 240]], dtype=np.int64)
    meas, scale = synth.poisson_counts(O.fpm_forward(obj, pupil, led)[0] ** 2, 1e3, rng, per_pixel=True)
    guess = (0.8 * obj * (1 + 0.3 * rng.standard_normal(obj.shape))).astype(np.complex64)
    check(fpm_sweep(cuda(guess), cuda(pupil), cuda(led), cuda(meas), scale),
          O.fpm_sweep(guess, pupil, led, meas, scale))


@pytest.mark.parametrize("ph, pw, count", [(16, 16, 1), (25, 16, 40), (20, 32, 3), (75, 64, 7), (18, 1024, 2),
                                           (250, 512, 3), (64, 128, 33)])
def test_subpixel_row_groups(ph, pw, count):
    from ptychox_b200.base import base_subpixel_sweep

    guess, probe, pos, meas, scale = problem(ph, pw, count, ph + pw, subpixel=True)
    check(base_subpixel_sweep(cuda(guess), cuda(probe), cuda(pos), cuda(meas), scale),
          O.base_subpix_sweep(guess, probe, pos, meas, scale))
