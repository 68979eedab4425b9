"""The amplitude of a photon count, ``sqrt(count * scale)``, as the sweeps' epilogues take it
(``ptx_counts.cuh``: a refined reciprocal square root) against CUDA's ``sqrtf`` of the rounded
product, value for value: every mantissa of a root's argument, and all 65536 counts at scales from
the smallest subnormal number to infinity."""

import shutil
import subprocess
from pathlib import Path

import pytest

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
