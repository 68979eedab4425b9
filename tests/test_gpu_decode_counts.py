"""The amplitude of a photon count, ``sqrt(count * scale)``, as the sweeps' epilogues take it
(``ptx_counts.cuh``: a refined reciprocal square root) against CUDA's ``sqrtf`` of the rounded
product, value for value: every mantissa of a root's argument, and all 65536 counts at scales from
the smallest subnormal number to infinity."""

import shutil
import subprocess
from pathlib import Path

import pytest
import torch

HERE = Path(__file__).resolve().parent
CSRC = HERE.parent / "ptychox_b200" / "csrc"


@pytest.mark.gpu
@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not on PATH")
def test_decoded_counts_are_the_square_roots(tmp_path):
    exe = tmp_path / "decode_counts"
    subprocess.run(["nvcc", "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", str(CSRC),
                    str(HERE / "decode_counts.cu"), "-o", str(exe)], check=True, capture_output=True, text=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    (mantissas, wrong), (counts, differing) = [[int(v) for v in line.split()] for line in out.splitlines()]
    assert mantissas == 1 << 24 and counts > 1000 * 65536
    assert wrong == 0
    assert differing == 0


@pytest.mark.gpu
@pytest.mark.parametrize("ph, pw, count, kind", [(64, 48, 3, "base"), (64, 40, 3, "base"), (64, 64, 2, "base"),
                                                 (96, 80, 2, "base"), (512, 32, 375, "base"), (64, 48, 2, "subpixel"),
                                                 (32, 32, 3, "fourier"), (24, 24, 3, "fourier")])
def test_sweeps_of_an_empty_object_scale_with_the_counts(ph, pw, count, kind):
    """Without light the loss is the mean of the squared amplitudes, and a factor of 4^k of the scale is
    one of 4^k of every value on the way (no sum comes near the ends of the range): the losses agree
    to the rounding of their FP64 sums, in the compilations for scales near and far from 1 alike."""
    from ptychox_b200.base import base_subpixel_sweep, base_sweep
    from ptychox_b200.fpm import fpm_sweep

    gen = torch.Generator(device="cuda").manual_seed(ph + pw)
    side = 128 if kind == "fourier" else max(ph, pw) + 8
    empty = torch.zeros(side, side, dtype=torch.complex64, device="cuda")
    aux = torch.randn(ph, pw, dtype=torch.complex64, generator=gen, device="cuda")
    pos = torch.randint(0, 9, (count, 2), generator=gen, device="cuda")
    counts = torch.randint(0, 200, (count, ph, pw), generator=gen, device="cuda").to(torch.int32).to(torch.uint16)
    sweep = {"base": base_sweep, "subpixel": base_subpixel_sweep, "fourier": fpm_sweep}[kind]
    pos = pos.double() if kind == "subpixel" else pos

    def loss(scale):
        return float(sweep(empty, aux, pos, counts, scale)[0])

    want = loss(1.3)
    assert abs(want - 1.3 * float(counts.to(torch.int64).double().mean())) <= 1e-6 * want
    for k in (-50, -33, -32, -31, 31, 32, 33, 50):
        assert abs(loss(1.3 * 4.0**k) / 4.0**k - want) <= 1e-12 * want
