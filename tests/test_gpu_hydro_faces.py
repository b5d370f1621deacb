"""FP64 face fluxes at the edges of their kernel's layout, against the oracle
bit for bit: rows around one and two 29-face warp segments, columns whose
length is not a multiple of the faces a thread marches over (grids above about
1e5 cells take more than one), the smallest grids, every boundary condition,
solver and limiter, both spatial orders."""
import dataclasses

import numpy as np
import pytest

import common  # noqa: F401  (paths)
import oracle
import torch_b200
from torch_b200 import config, workloads

pytestmark = pytest.mark.gpu

SIZES = [(3, 1, 1), (28, 1, 1), (29, 1, 1), (58, 1, 1), (5, 3, 1), (57, 33, 1), (4, 3, 5), (30, 7, 6)]
BOUNDARIES = ["outflow", "reflecting", "periodic", "inflow", "free"]


def case(ncells, riemann, limiter, boundary, order):
    """Random states: density and pressure over a decade, velocities around
    the sound speed, ionisation and advected fractions."""
    nx, ny, nz = ncells
    nd = 1 if ny == 1 else (2 if nz == 1 else 3)
    tp = workloads.sedov_parameters(n=nx, nd=nd, order=order, riemann=riemann, limiter=limiter)
    tp = dataclasses.replace(tp, ncells=ncells, leftBC=(boundary,) * 3, rightBC=(boundary,) * 3,
                             star_position=(0, 0, 0))
    rng = np.random.default_rng(nx + 100 * ny + 1000 * nz)
    n = nx * ny * nz
    den, pre = 1e-20 * 10 ** rng.uniform(-0.5, 0.5, n), 1e-10 * 10 ** rng.uniform(-0.5, 0.5, n)
    vel = 1e5 * rng.standard_normal((3, n))
    vel[:, rng.random(n) < 0.2] = 0.0  # no jump, and jumps along or across one axis
    vel[1:, rng.random(n) < 0.2] = 0.0
    vel[nd:] = 0.0
    ic = config.make_initial_conditions(ncells, tp.sideLength / nx, den, pre, rng.random(n), vel)
    return tp, ic


def check(tp, ic, steps):
    t, o = torch_b200.Torch(tp, ic), oracle.Oracle(tp, ic)
    dts = t.run_steps(steps)
    ref_dts = [o.full_step() for _ in range(steps)]
    got, ref = t.state().U, o.state().U
    t.close()
    assert np.array_equal(dts, np.array(ref_dts))
    assert np.array_equal(got[:4 + ic.nd], ref.reshape(got.shape)[:4 + ic.nd])


@pytest.mark.parametrize("ncells", SIZES)
@pytest.mark.parametrize("boundary", BOUNDARIES)
def test_faces_bitwise_at_layout_edges(ncells, boundary):
    order = 0 if ncells[0] == 4 else 1
    check(*case(ncells, "RotatedHLLC", "albada", boundary, order), steps=4)


@pytest.mark.parametrize("riemann", ["HLL", "HLLC", "RotatedHLLC"])
@pytest.mark.parametrize("limiter", ["minmod", "superbee", "albada"])
def test_faces_bitwise_solvers_and_limiters(riemann, limiter):
    check(*case((30, 7, 6), riemann, limiter, "outflow", 1), steps=4)


@pytest.mark.parametrize("ncells", [(71, 61, 33), (350, 353, 1)])
def test_faces_bitwise_marched_columns(ncells):
    check(*case(ncells, "RotatedHLLC", "albada", "reflecting", 1), steps=3)
