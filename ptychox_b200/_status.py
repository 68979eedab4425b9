"""Device-side window checks of the conventional operators, reported without a host sync.

The conventional kernels check every scan window on the device: a window that leaves the
object is skipped and bit 0 of the workspace status word is set (``ptx_workspace_status``).
Positions that arrive as host tensors are checked on the host before the launch (no device
round trip).  For device-resident positions -- the reference's training loop indexes a
device tensor of positions every step (``train_ptychography.py:549``) -- three modes:

* ``"deferred"`` (default): after the launch the status word is copied in stream order into a
  page-locked slot and an event is recorded; the next call of any conventional operator on
  that device (or :func:`check_errors`) raises ``ValueError`` for every earlier call whose
  copy has completed with the bit set.  No host synchronisation, no host copy of positions.
* ``"sync"``: the same copy, waited for at once, so the offending call itself raises.
* ``"host"``: the positions are copied to the host and checked before the launch (one
  device-to-host synchronisation per call).

The same word tells of a device wait of the sweep that gave up (bit 1: its loss and gradients are
NaN), which is raised as ``PtychoXError`` where the call is retired.

Calls made while a stream is being captured into a CUDA graph are not tracked.
"""

from __future__ import annotations

import ctypes

import torch

from . import _abi
from ._utils import stream_handle

_MODES = ("deferred", "sync", "host")
_mode = "deferred"
_calls: list[str] = []  # names of the tracked operators; a tracked call's tag is its index here
_tags: dict[str, int] = {}


def set_bounds_check(mode: str) -> None:
    """Select how out-of-object windows of device-resident positions are reported:
    ``"deferred"`` (default), ``"sync"`` or ``"host"`` (see the module docstring)."""
    global _mode
    if mode not in _MODES:
        raise ValueError(f"bounds check mode must be one of {_MODES}, got {mode!r}")
    _mode = mode


def bounds_check_mode() -> str:
    return _mode


def _raise_for(what: str) -> None:
    raise ValueError(f"{what}: a scan window leaves the object (its frame was skipped); "
                     "positions must satisfy 0 <= x <= W - pw and 0 <= y <= H - ph.")


def _poll(device: int, block: bool) -> None:
    """Retire tracked calls of `device` (all when negative); raise for the first failure."""
    if not _calls:
        return
    failed = ctypes.c_int(-1)
    _abi.call("ptx_status_poll", device, int(block), failed)
    if failed.value >= 0:
        _raise_for(_calls[failed.value])


def check_errors(block: bool = True) -> None:
    """Raise ``ValueError`` if an earlier conventional call with device positions met a window
    outside the object (waits for their status copies when ``block``)."""
    _poll(-1, block)


def before_call(device: torch.device) -> None:
    """Report completed failures of earlier calls on `device` (non-blocking)."""
    if _calls and device.index is not None:
        _poll(device.index, False)


def after_call(workspace: torch.Tensor, device: torch.device, what: str) -> None:
    """Queue the status copy of the call that just used `workspace` (device positions only);
    `device` is current."""
    tag = _tags.get(what)
    if tag is None:
        _calls.append(what)
        tag = _tags[what] = _calls.index(what)
    failed = ctypes.c_int(-1)
    _abi.call("ptx_status_track", workspace.data_ptr(), tag, failed, stream_handle(device))
    if failed.value >= 0:
        _raise_for(_calls[failed.value])
    if _mode == "sync":
        _poll(device.index if device.index is not None else torch.cuda.current_device(), True)
