"""Coded sweeps and adjoints whose gradients are written over an argument that is read no more by
then: the object gradient leaves with the last launch, so it may take the place of any input, and the
finite-difference sweep reads the object before it clears the coded-surface gradient.  The results
are those of separate buffers, but for the order of the float atomics: compared at 1e-5 relative L2,
the tolerance of the oracle tests."""

import numpy as np
import pytest
import torch

from conftest import rel_l2
from oracle import ptycho_oracle as O

pytestmark = pytest.mark.gpu

COUNT, DS = 5, 2


def cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def problem(n):
    from ptychox_b200 import synth

    rng = np.random.default_rng(n)
    obj, mask = synth.random_object(n, n, rng), synth.binary_mask(n, 0.5, rng)
    t1 = synth.angular_spectrum_transfer(n, 1.85e-6, 0.5e-6, 396.95e-6)
    t2 = synth.angular_spectrum_transfer(n, 1.85e-6, 0.5e-6, 2e-3)
    shifts = synth.coded_shifts(COUNT, 5.0, n, rng).astype(np.float32)
    return rng, obj, mask, t1, t2, shifts


def gradient_over(buffers, name, n, place):
    """(object gradient, coded-surface gradient, buffers) with `place` of the two over buffer `name`
    (made as large as a field)."""
    if name is not None and buffers[name].numel() * buffers[name].element_size() < 8 * n * n:
        t = buffers[name]
        room = torch.zeros(8 * n * n // t.element_size(), dtype=t.dtype, device="cuda")
        room[:t.numel()] = t.reshape(-1)
        buffers[name] = room
    grads = {p: torch.empty(8 * n * n, dtype=torch.uint8, device="cuda") for p in ("object", "coded")}
    if name is not None:
        grads[place] = buffers[name].reshape(-1).view(torch.uint8)[:8 * n * n]
    return grads


def field(raw, n):
    return raw.view(torch.complex64).reshape(n, n).cpu().numpy()


@pytest.mark.parametrize("n", [64, 60])
@pytest.mark.parametrize("over", ["grad_output", "x_forward", "sensor", "amplitude", "transfer_1", "transfer_2",
                                  "coded_surface", "shifts"])
def test_adjoint(n, over):
    from ptychox_b200 import _abi
    from ptychox_b200._utils import call_on, workspace

    rng, obj, mask, t1, t2, shifts = problem(n)
    _, xf, sensor, amp = O.coded_forward(obj, mask, t1, t2, shifts, DS)
    gout = rng.standard_normal(amp.shape).astype(np.float32)
    dev = torch.device("cuda", torch.cuda.current_device())

    def run(name):
        t = {"grad_output": gout, "x_forward": xf.astype(np.complex64), "sensor": sensor.astype(np.complex64),
             "amplitude": amp.astype(np.float32), "coded_surface": mask, "transfer_1": t1, "transfer_2": t2,
             "shifts": shifts}
        t = {k: cuda(v) for k, v in t.items()}
        g = gradient_over(t, name, n, "object")
        ws = workspace(_abi.query("ptx_coded_workspace_bytes", n, COUNT), dev)
        call_on(dev, "ptx_coded_backward", *(t[k].data_ptr() for k in (
            "grad_output", "x_forward", "sensor", "amplitude", "coded_surface", "transfer_1", "transfer_2")), n,
            t["shifts"].data_ptr(), COUNT, DS, g["object"].data_ptr(), g["coded"].data_ptr(), ws.data_ptr(), ws.numel())
        return field(g["object"], n), field(g["coded"], n)

    for got, want in zip(run(over), run(None)):
        assert rel_l2(got, want) < 1e-5


@pytest.mark.parametrize("n", [64, 60])
@pytest.mark.parametrize("loss, place, over", [
    *(("mse", "object", name) for name in ("object", "coded_surface", "transfer_1", "transfer_2", "shifts", "measured")),
    *(("fd", "object", name) for name in ("object", "coded_surface", "transfer_1", "transfer_2", "shifts", "measured")),
    ("fd", "coded", "object"),
])
def test_sweep(n, loss, place, over):
    from ptychox_b200 import _abi, synth
    from ptychox_b200._utils import call_on, workspace

    rng, obj, mask, t1, t2, shifts = problem(n)
    amp = O.coded_forward(obj, mask, t1, t2, shifts, DS)[3]
    meas, scale = synth.poisson_counts(amp**2, 1e3, rng, per_pixel=True)
    guess = (0.8 * obj * (1 + 0.3 * rng.standard_normal(obj.shape))).astype(np.complex64)
    dev = torch.device("cuda", torch.cuda.current_device())

    def run(name):
        t = {k: cuda(v) for k, v in {"object": guess, "coded_surface": mask, "transfer_1": t1, "transfer_2": t2,
                                     "shifts": shifts, "measured": meas}.items()}
        g = gradient_over(t, name, n, place)
        value = torch.empty((), dtype=torch.float64, device=dev)
        fields = [t[k].data_ptr() for k in ("object", "coded_surface", "transfer_1", "transfer_2")]
        call = [*fields, n, t["shifts"].data_ptr(), COUNT, DS, t["measured"].data_ptr(), scale]
        out = [value.data_ptr(), g["object"].data_ptr(), g["coded"].data_ptr()]
        if loss == "mse":
            ws = workspace(_abi.query("ptx_coded_workspace_bytes", n, COUNT), dev)
            call_on(dev, "ptx_coded_sweep", *call, *out, ws.data_ptr(), ws.numel())
        else:
            ws = workspace(_abi.query("ptx_coded_sweep_ex_workspace_bytes", n, COUNT, DS, 1), dev)
            shift_grad = torch.empty(COUNT, 2, dtype=torch.float64, device=dev)
            call_on(dev, "ptx_coded_sweep_ex", *call, 1, *out, shift_grad.data_ptr(), ws.data_ptr(), ws.numel())
        return field(g["object"], n), field(g["coded"], n), value.cpu().numpy()

    for got, want in zip(run(over), run(None)):
        assert rel_l2(got, want) < 1e-5
