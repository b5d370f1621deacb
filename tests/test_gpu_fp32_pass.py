"""The FP32 hydro pass where its tiling and its shortened divisions can go
wrong: every depth of the z chunks (ragged last chunks, more CTAs than fit at
once) leaves the same bits, and velocity differences whose squares are
subnormal leave a finite state that follows the FP64 form."""
import dataclasses

import numpy as np
import pytest

import common
import torch_b200
from torch_b200 import workloads

pytestmark = pytest.mark.gpu


def run(tp, ic, steps, precision, depth=None):
    t = torch_b200.Torch(tp, ic, precision=precision)
    if depth:
        t.set_tile(depth)
    t.run_steps(steps)
    s = t.state()
    t.close()
    return s


@pytest.mark.parametrize("kind,n", [("sedov", 33), ("sedov", 100), ("hii", 75)])
def test_depth_of_the_chunks_keeps_every_bit(kind, n):
    tp, ic = workloads.sedov(n=n) if kind == "sedov" else workloads.hii_region(n=n, seed=2)
    ref = run(tp, ic, 4, torch_b200.PRECISION_FP32)
    for depth in (1, 7, 17, n):
        got = run(tp, ic, 4, torch_b200.PRECISION_FP32, depth)
        assert np.array_equal(got.U, ref.U), depth


@pytest.mark.parametrize("limiter", ["albada", "leer"])
@pytest.mark.parametrize("size", [1e-16, 1e-19, 1e-21])
def test_subnormal_squares_of_differences(limiter, size):
    """Gas with velocities of `size` sound speeds, in code units whose limiter
    cut lies below the smallest normal number.  The FP32 form's error is that
    of the blast-wave comparison (1e-5)."""
    tp, ic = workloads.sedov(n=24, limiter=limiter)
    tp = dataclasses.replace(tp, pscale=1.0e-26)
    rng = np.random.default_rng(7)
    c = np.sqrt(np.median(ic.pre) / np.median(ic.den))
    for d in range(3):
        ic.vel[d] = rng.normal(0, size * c, ic.den.size)
    a = run(tp, ic, 6, torch_b200.PRECISION_FP32)
    b = run(tp, ic, 6, torch_b200.PRECISION_FP64)
    assert np.isfinite(a.U).all()
    assert common.rel_l1(a.U[0], b.U[0]) <= 1e-5 and common.rel_l1(a.U[1], b.U[1]) <= 1e-5
