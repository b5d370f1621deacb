"""Sweeps at the limit of what one CTA can walk (its shared memory holds a ring
of three shells and every shell's offset), run for real: the last size that
fits and one that does not, against the oracle, and a batch whose grids fit
only one by one, against the grids alone."""
import dataclasses

import numpy as np
import pytest

import common
import known_answers
import oracle
import torch_b200
from torch_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [57000, 60000])
def test_sweeps_of_very_many_shells(cells):
    tp, ic = known_answers.spitzer_case(cells, 6.0)
    t, o = torch_b200.Torch(tp, ic), oracle.Oracle(tp, ic)
    t.run_steps(4)
    for _ in range(4):
        o.full_step()
    got, ref = t.state(), o.state()
    t.close()
    for f in ("U", "R", "T"):
        a, b = getattr(got, f), getattr(ref, f)
        for row in range(a.shape[0]):
            if common.inplane(f, row, 1):
                assert common.rel_l1(a[row], b[row]) <= 1e-10, (f, row)
    assert np.all(got.R[1][2:] > 0) and np.all(got.T[0][2:] > 0)  # optical depths and column densities


def test_batch_of_a_long_and_a_wide_grid():
    def grid(nx, ny, **kw):
        tp, ic = workloads.blister((nx, ny, 1), **kw)
        # gas in motion, so that every step's column densities are others
        ic.vel[:2] = 1e6 * np.random.default_rng(nx).standard_normal((2, nx * ny))
        return dataclasses.replace(tp, windCellRadius=0, massLossRate=0.0), ic

    cases = [grid(50000, 3, side=0.5 * workloads.PC2CM), grid(500, 1000)]
    grids = [torch_b200.Torch(tp, ic) for tp, ic in cases]
    dt_next = min(g.dt_max for g in grids)
    b = torch_b200.Batch(grids)
    b.run_steps(5, dt_next)
    got = [g.state() for g in grids]
    b.close()
    for (tp, ic), g, s in zip(cases, grids, got):
        g.close()
        t = torch_b200.Torch(tp, ic)
        t.run_steps(5, dt_next)
        ref = t.state()
        t.close()
        for f in ("U", "Q", "R", "T"):
            assert np.array_equal(getattr(s, f), getattr(ref, f)), f
