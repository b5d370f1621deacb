"""Passes that leave out what cannot change, against the general ones: the
FP32 form's radiation and thermal updates (the thermal one and the heating
pass run in their general form while the heating terms are kept), states the
host sets outside the floors, and the time-step reduction with many cells per
thread against one cell per thread (as it runs while conservation sums are
recorded)."""
import dataclasses

import numpy as np
import pytest

import common  # noqa: F401  (paths)
import torch_b200
from torch_b200 import workloads

pytestmark = pytest.mark.gpu
FORMS = [torch_b200.PRECISION_FP64, torch_b200.PRECISION_FP32]


def run(tp, ic, form, steps, setup=None):
    t = torch_b200.Torch(tp, ic, precision=form)
    if setup:
        setup(t)
    dts = t.run_steps(steps)
    s = t.state()
    t.close()
    return dts, s


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("case", ["hii", "blister", "tti"])
def test_lean_passes_equal_general_ones(form, case):
    if case == "hii":
        tp, ic = workloads.hii_region(n=20, seed=9)
    else:
        tp, ic = workloads.blister((45, 60, 1))
        if case == "tti":
            tp = dataclasses.replace(tp, rt_coupling="tti")
    dts, got = run(tp, ic, form, 10)
    ref_dts, ref = run(tp, ic, form, 10, lambda t: t.heating_enable(True))
    # one rounding per update apart in the FP32 form, the same values in the FP64 form
    tol = 0 if form == torch_b200.PRECISION_FP64 else 1e-10
    assert np.allclose(dts, ref_dts, rtol=tol, atol=0)
    for f in ("U", "Q", "R", "T"):
        a, b = getattr(got, f), getattr(ref, f)
        scale = np.abs(b).max(axis=1, keepdims=True) + 1e-300
        assert np.all(np.abs(a - b) <= tol * scale), f


@pytest.mark.parametrize("form", FORMS)
def test_state_set_outside_the_floors_is_fixed(form):
    """Energy below the kinetic energy, fractions above 1, set by the host in
    the middle of a run: the first update of the next step fixes every cell."""
    tp, ic = workloads.hii_region(n=16, seed=4)
    t = torch_b200.Torch(tp, ic, precision=form)
    t.run_steps(5)
    U = t.state().U
    U[1, 100:140] *= 1e-12
    U[2, 200:260] = 1.5 * U[0, 200:260]
    U[3, 300:330] = -U[0, 300:330]
    t.set_conserved(U)
    t.run_steps(1)
    V = t.state().U
    t.close()
    ke = (V[4:] ** 2).sum(axis=0) / (2 * V[0])
    assert np.all(np.isfinite(V)) and np.all(V[1] - ke > 0)
    assert np.all(V[2] <= V[0] * (1 + 1e-12)) and np.all(V[3] >= 0)


@pytest.mark.parametrize("form", FORMS)
def test_time_step_with_many_cells_per_thread(form):
    tp, ic = workloads.hii_region(n=70, seed=3)
    dts, got = run(tp, ic, form, 4)
    ref_dts, ref = run(tp, ic, form, 4, lambda t: t.conservation_enable(True))
    assert np.array_equal(dts, ref_dts) and np.array_equal(got.U, ref.U)


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("case", ["hydro_2d", "hydro_3d", "hii"])
def test_overlapped_launches_equal_serial_ones(monkeypatch, form, case):
    """Kernels launched while the one before them still runs wait for it before
    they read anything (TRG_SHELL_OVERLAP=0 launches them one after another)."""
    if case == "hii":
        tp, ic = workloads.hii_region(n=24, seed=8)
    elif case == "hydro_2d":
        tp, ic = workloads.blister()
        tp = dataclasses.replace(tp, radiation_on=False, cooling_on=False)
    else:
        tp, ic = workloads.sedov(n=40)
    dts, got = run(tp, ic, form, 30)
    monkeypatch.setenv("TRG_SHELL_OVERLAP", "0")
    ref_dts, ref = run(tp, ic, form, 30)
    assert np.array_equal(dts, ref_dts) and np.array_equal(got.U, ref.U) and np.array_equal(got.Q, ref.Q)
