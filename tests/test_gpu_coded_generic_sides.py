"""Coded and near-field sweeps at large mixed-radix field sides that no other test visits, with the
shift gradient, against the FP64 oracle.  Tolerance: relative L2 below 1e-5, or five times the error
of the oracle's complex64 formulation where that misses it, as in the tests of the passes."""

import pytest

from test_gpu_coded_passes import check, cuda, problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, ds, nearfield", [(648, 2, True), (675, 5, False), (720, 4, True), (729, 3, True),
                                              (750, 2, False), (750, 2, True), (768, 4, False), (800, 5, True),
                                              (810, 2, True), (864, 4, True), (900, 2, False)])
def test_sweep(n, ds, nearfield):
    from ptychox_b200.coded import coded_sweep

    args = problem(n, 2, ds, nearfield)
    guess, mask, t1, t2, shifts, meas, scale = args
    got = coded_sweep(cuda(guess), cuda(mask), cuda(t1), cuda(t2), cuda(shifts), ds, cuda(meas), scale, with_shifts=True)
    check(got, args, ds)
