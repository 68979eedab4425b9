"""The 512-point column pipeline where it is taken: five tiles or more per CTA, so that every CTA's
buffers and barriers come round, at one tile below and around whole rounds of CTAs, with narrow and
wide frames, and in the sub-pixel and the Fourier sweep.  Against the FP64 oracle, relative L2 below
1e-5 as in the other tests of the passes."""

import numpy as np
import pytest
import torch

from oracle import ptycho_oracle as O
from test_gpu_pass_pipeline import check, cuda, problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pw, count", [(32, 369), (32, 370), (32, 371), (64, 185), (96, 124), (512, 24)])
def test_column_pipeline(pw, count):
    from ptychox_b200.base import base_sweep

    guess, probe, pos, meas, scale = problem(512, pw, count, pw + count)
    check(base_sweep(cuda(guess), cuda(probe), cuda(pos), cuda(meas), scale), O.base_sweep(guess, probe, pos, meas, scale))


def test_column_pipeline_of_the_subpixel_sweep():
    from ptychox_b200.base import base_subpixel_sweep

    guess, probe, pos, meas, scale = problem(512, 32, 372, 5, subpixel=True)
    check(base_subpixel_sweep(cuda(guess), cuda(probe), cuda(pos), cuda(meas), scale),
          O.base_subpix_sweep(guess, probe, pos, meas, scale))


def test_column_pipeline_of_the_fourier_sweep():
    from ptychox_b200 import synth
    from ptychox_b200.fpm import fpm_sweep

    rng = np.random.default_rng(4)
    obj, pupil = synth.random_object(1024, 1024, rng), synth.circular_pupil(512, 0.3)
    led = rng.integers(200, 312, size=(25, 2)).astype(np.int64)
    meas, scale = synth.poisson_counts(O.fpm_forward(obj, pupil, led)[0] ** 2, 1e3, rng, per_pixel=True)
    guess = (0.8 * obj * (1 + 0.3 * rng.standard_normal(obj.shape))).astype(np.complex64)
    check(fpm_sweep(cuda(guess), cuda(pupil), cuda(led), cuda(meas), scale),
          O.fpm_sweep(guess, pupil, led, meas, scale))
