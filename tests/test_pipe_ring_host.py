"""Waits of the 512-point column pipeline over every order in which its copies can complete.

``PipeRing`` (``ptx_pipering.h``) names each tile's group of threads, buffer, barrier and phase.
``pipe_ring_host.cpp`` walks all interleavings of the two groups and their copies on the host: no
wait may return before its own tile has come, no copy may be issued into a buffer or on a barrier
still in use, every schedule has to come to its end, and a CTA that gives up on a copy knows which
copies it still has under way.
"""
import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent
CSRC = HERE.parent / "ptychox_b200" / "csrc"


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ not on PATH")
def test_no_wait_returns_before_its_tile(tmp_path):
    exe = tmp_path / "pipe_ring_host"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", str(CSRC), str(HERE / "pipe_ring_host.cpp"), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    rows = [[int(v) for v in line.split()] for line in out.splitlines()]
    assert [r[0] for r in rows] == list(range(1, 21))
    for n, states, early, in_use, stuck, wrong_open in rows:
        assert states > n
        assert (early, in_use, stuck, wrong_open) == (0, 0, 0, 0), n


def test_status_word_codes():
    """Bit 0: a window outside the object; bit 1: a device wait that gave up."""
    from ptychox_b200 import _abi
    from ptychox_b200.build import build_library

    build_library()
    codes = [_abi.query("ptx_status_code", word) for word in range(4)]
    assert codes == [_abi.PTX_OK, _abi.PTX_ERR_OUT_OF_BOUNDS, _abi.PTX_ERR_TIMEOUT, _abi.PTX_ERR_OUT_OF_BOUNDS]
