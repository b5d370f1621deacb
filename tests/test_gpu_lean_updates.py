"""The FP32 form's lean radiation and thermal updates in 3-D grids against the
general ones."""
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
