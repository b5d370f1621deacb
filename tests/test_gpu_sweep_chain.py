"""Causal sweeps walked by one CTA against the same sweeps launched shell by
shell (TRG_SHELL_OVERLAP=0): bit for bit in the exact build, to rounding in
the fast one.  Sizes: one cell per shell, shells of one more cell than a
group has threads, shells of several cells per thread, a wind that empties
the first shells, stars in a corner and beside an edge, 3-D grids with the
chain for both sweeps and for the column densities alone."""
import dataclasses

import numpy as np
import pytest

import common  # noqa: F401  (paths)
import known_answers
import torch_b200
from torch_b200 import config, workloads

pytestmark = pytest.mark.gpu


def blister(nx, ny, star_y=None, wind=0):
    tp, ic = workloads.blister((nx, ny, 1), star_cell_y=star_y)
    return dataclasses.replace(tp, windCellRadius=wind, massLossRate=tp.massLossRate if wind else 0.0), ic


def hii(n, star):
    tp, ic = workloads.hii_region(n=n, seed=5)
    return dataclasses.replace(tp, star_position=star), ic


CASES = {
    "1d": lambda: known_answers.spitzer_case(200, 6.0),
    "2d_small": lambda: blister(7, 5),
    "2d_wind": lambda: blister(40, 53, wind=6),
    "2d_257_cells": lambda: blister(129, 40),
    "2d_many_per_thread": lambda: blister(420, 96),
    "2d_corner": lambda: blister(33, 70, star_y=0),
    "3d_centre": lambda: hii(12, (6, 6, 6)),
    "3d_corner": lambda: hii(11, (0, 0, 10)),
    "3d_column_density_only": lambda: hii(17, (8, 8, 8)),
}


def steps(tp, ic, form, n):
    t = torch_b200.Torch(tp, ic, precision=form)
    dts = t.run_steps(n)
    s = t.state()
    t.close()
    return dts, s


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("form", [torch_b200.PRECISION_FP64, torch_b200.PRECISION_FP32])
def test_chain_equals_shell_launches(monkeypatch, name, form):
    tp, ic = CASES[name]()
    if form == torch_b200.PRECISION_FP32 and ic.nd == 1:
        pytest.skip("the FP32 form needs a 2-D or 3-D grid")
    monkeypatch.setenv("TRG_SHELL_OVERLAP", "0")
    ref_dts, ref = steps(tp, ic, form, 9)
    monkeypatch.delenv("TRG_SHELL_OVERLAP")
    dts, got = steps(tp, ic, form, 9)
    for f in ("U", "Q", "R", "T"):
        a, b = getattr(got, f), getattr(ref, f)
        if form == torch_b200.PRECISION_FP64:
            assert np.array_equal(a, b, equal_nan=True), f
        else:
            scale = np.abs(b).max(axis=1, keepdims=True) + 1e-300
            assert np.all(np.abs(a - b) <= 1e-11 * scale), f
    assert np.allclose(dts, ref_dts, rtol=0 if form == torch_b200.PRECISION_FP64 else 1e-11, atol=0)


@pytest.mark.parametrize("sizes", [[(20, 33), (61, 17)], [(30, 40), (420, 96), (9, 12)]])
def test_batched_chains_equal_single_grids(sizes):
    """One CTA per grid of a batch, its threads set by the largest grid."""
    cases = [blister(nx, ny) for nx, ny in sizes]
    grids = [torch_b200.Torch(tp, ic) for tp, ic in cases]
    dt_next = min(g.dt_max for g in grids)
    b = torch_b200.Batch(grids)
    b.run_steps(7, dt_next)
    got = [g.state() for g in grids]
    b.close()
    for (tp, ic), g, s in zip(cases, grids, got):
        g.close()
        t = torch_b200.Torch(tp, ic)
        t.run_steps(7, dt_next)
        ref = t.state()
        t.close()
        for f in ("U", "Q", "R", "T"):
            assert np.array_equal(getattr(s, f), getattr(ref, f)), f


@pytest.mark.parametrize("form", [torch_b200.PRECISION_FP64, torch_b200.PRECISION_FP32])
def test_tied_axes_read_no_cell_of_their_own_shell(monkeypatch, form):
    """A star in a cell's centre: on the diagonals two axes tie, and a neighbour
    level with the cell belongs to the cell's own shell.  Its weight is exactly
    0 in both builds (49 times the rounded 1/49 is not 1), or the chain would be
    refused and the sweeps launched shell by shell (two times 65 launches)."""
    n = 131
    tp = workloads.hii_region_parameters(n=n)
    tp = dataclasses.replace(tp, nd=2, ncells=(n, n, 1), star_position=(65, 65, 0))
    rng = np.random.default_rng(2)
    den = 1e3 * workloads.setups.HYDROGEN_MASS * np.exp(0.3 * rng.standard_normal(n * n))
    ic = config.make_initial_conditions((n, n, 1), tp.sideLength / n, den,
                                        den * workloads.setups.SPECIFIC_GAS_CONSTANT * 100.0, np.zeros(n * n),
                                        np.zeros((3, n * n)))
    t = torch_b200.Torch(tp, ic, precision=form)
    before = t.kernel_launches()
    t.run_steps(6)
    launches = t.kernel_launches() - before
    got = t.state()
    t.close()
    assert launches < 6 * 60
    monkeypatch.setenv("TRG_SHELL_OVERLAP", "0")
    _, ref = steps(tp, ic, form, 6)
    scale = np.abs(ref.U).max(axis=1, keepdims=True) + 1e-300
    assert np.all(np.abs(got.U - ref.U) <= (0 if form == torch_b200.PRECISION_FP64 else 1e-11) * scale)
