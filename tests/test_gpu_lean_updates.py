"""The FP32 form's lean radiation and thermal updates in 3-D grids against the
general ones.

A state that the host has set takes the general update in the first sub-step of
the next step.  So each of some consecutive steps, which begin with radiation,
hydrodynamics and cooling in turn, is taken twice from the same state: by the
run itself, and by a second context whose state is set anew."""
import dataclasses

import numpy as np
import pytest

import common  # noqa: F401  (paths)
import torch_b200
from torch_b200 import workloads

pytestmark = pytest.mark.gpu
T_HEAT = common.FIELD_NAMES["T"].index("heat")


@pytest.mark.parametrize("queue", [0, 1])
@pytest.mark.parametrize("subcycling", [True, False])
def test_heating_rate_is_cleared_in_cells_that_fall_below_the_switch(queue, subcycling):
    """A thermal sub-step clears the heating rate of every cell outside the
    wind.  Cells whose ADV the hydro sub-step carries below the HII switch
    between the step's rates and its thermal sub-step are among them."""
    n = 24
    tp, ic = workloads.hii_region(n=n, seed=6)
    tp = dataclasses.replace(tp, star_on=subcycling, thermoSubcycling=subcycling)
    t = torch_b200.Torch(tp, ic, precision=torch_b200.PRECISION_FP32)
    if queue:
        t.thermo_queue(2)
    t.run_steps(8)
    s = t.state()
    U, neutral = s.U, s.Q[2] < 1e-3
    x = np.arange(n ** 3) % n
    # gas just above the switch streams out of slabs into which gas below it follows
    adv = np.where(x % 6 < 3, np.where(x < n // 2, 1.0, 1.002 * tp.thermoHII_Switch), 0.0)
    U[3] = np.where(neutral, adv, 1.0) * U[0]
    speed = 0.4 * np.sqrt(U[1] / U[0])
    U[1] += 0.5 * U[0] * speed ** 2
    U[4] += U[0] * speed
    t.set_conserved(U)
    below = above = 0
    for _ in range(9):
        before = t.state().Q[3] >= tp.thermoHII_Switch
        t.run_steps(1)
        s = t.state()
        now = s.Q[3] >= tp.thermoHII_Switch
        below += int((before & ~now).sum())
        above += int(now.sum())
        assert np.all(s.T[T_HEAT] == 0), np.count_nonzero(s.T[T_HEAT])
    t.close()
    assert below > 100 and above > 1000  # cells did cross the switch


def grids(case, n=24):
    tp, ic = workloads.hii_region(n=n, seed=9)
    if case == "wind":  # cells of a wind, and gas that it drives
        tp = dataclasses.replace(tp, windCellRadius=3, massLossRate=1e20, windVelocity=3e6)
    elif case == "floors":  # neutral gas at the temperature floor, cooling gas that reaches it
        tp = dataclasses.replace(tp, tfloor=200.0, pfloor=3e-11)
    elif case == "no_subcycling":
        tp = dataclasses.replace(tp, thermoSubcycling=False)
    elif case == "constants":
        tp = dataclasses.replace(tp, K4=0.3, massFractionH=0.7, heatCapacityRatio=1.4)
    return tp, ic


@pytest.mark.parametrize("case", ["plain", "wind", "floors", "no_subcycling", "constants", "queue", "switch"])
def test_steps_with_lean_updates_equal_steps_with_general_ones(case):
    """The two differ by roundings of the first sub-step's FP64 update (a few
    2^-53).  Such a difference tips a rounding of the FP32 hydro pass, by at
    most 2^-24 of a cell's fluxes, in about one of 2^29 roundings: no cell is
    off by more than 1e-7 of its field's largest value, and the fields' relative
    L1 difference is that of a few tipped roundings in 24^3 cells at most."""
    tp, ic = grids(case)
    n = ic.ncells[0]
    t, general = (torch_b200.Torch(tp, ic, precision=torch_b200.PRECISION_FP32) for _ in range(2))
    if case == "queue":
        t.thermo_queue(2)
        general.thermo_queue(2)
    t.run_steps(12)
    if case == "switch":  # neutral gas above, at and below the HII switch, in motion
        s = t.state()
        x = np.arange(n ** 3) % n
        adv = np.choose(x % 6 // 2, [0.0, 1.01 * tp.thermoHII_Switch, 1.0])
        s.U[3] = np.where(s.Q[2] < 1e-3, adv, 1.0) * s.U[0]
        speed = 0.3 * np.sqrt(s.U[1] / s.U[0])
        s.U[1] += 0.5 * s.U[0] * speed ** 2
        s.U[4] += s.U[0] * speed
        t.set_conserved(s.U)
        t.run_steps(1)
    for k in range(6):
        general.restore(t.checkpoint())
        general.set_conserved(general.state().U)
        assert np.isclose(t.run_steps(1)[0], general.run_steps(1)[0], rtol=1e-12, atol=0)
        got, ref = t.state(), general.state()
        for g in ("U", "Q", "R", "T"):
            for row, name in enumerate(common.FIELD_NAMES[g]):
                a, b = getattr(got, g)[row], getattr(ref, g)[row]
                what = (k, g, name)
                assert np.all(np.abs(a - b) <= 1e-7 * np.abs(b).max()), what
                # (HEAT is what is left of heating and cooling that cancel)
                assert common.rel_l1(a, b) <= (1e-8 if name == "heat" else 1e-10), what
    t.close()
    general.close()
