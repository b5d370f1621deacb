"""What the library launches and reports, on a CUDA runtime that runs nothing
(fake_gpu)."""
import dataclasses
import struct

import numpy as np
import pytest

import fake_gpu
import known_answers
import torch_b200
from torch_b200 import workloads

FP64, FP32 = torch_b200.PRECISION_FP64, torch_b200.PRECISION_FP32


@pytest.fixture
def gpu():
    with fake_gpu.fake_gpu() as g:
        yield g


def blister(nx=40, ny=53, wind=0):
    tp, ic = workloads.blister((nx, ny, 1))
    return dataclasses.replace(tp, windCellRadius=wind, massLossRate=tp.massLossRate if wind else 0.0), ic


# --------------------------------------------------------- refused launches
CASES = {
    "spitzer_1d": (lambda: known_answers.spitzer_case(60, 6.0), FP64),
    "blister_fp64": (blister, FP64),
    "blister_fp32": (blister, FP32),
    "hii_fp32": (lambda: workloads.hii_region(n=24, seed=1), FP32),
    "sedov_fp64": (lambda: workloads.sedov(n=12), FP64),
    "sedov_fp32": (lambda: workloads.sedov(n=12), FP32),
}


def kernels(gpu):
    return sorted({l.name for l in gpu.launches()})


@pytest.mark.parametrize("case", sorted(CASES))
def test_refused_launches_are_reported(gpu, case):
    """Whichever kernel of a run the runtime refuses to launch, in a captured
    sweep or not: the call that needs it fails."""
    make, form = CASES[case]
    tp, ic = make()
    t = torch_b200.Torch(tp, ic, precision=form)
    created = kernels(gpu)
    gpu.reset()
    t.run_steps(6)
    stepped = kernels(gpu)
    t.close()
    assert len(stepped) > 2
    for name in created:
        gpu.reset()
        gpu.refuse(name)
        with pytest.raises(torch_b200.TrgError):
            torch_b200.Torch(tp, ic, precision=form)
        assert gpu.counts()["refused"], name
    for name in stepped:
        gpu.reset()
        t = torch_b200.Torch(tp, ic, precision=form)
        gpu.refuse(name)
        with pytest.raises(torch_b200.TrgError):
            t.run_steps(6)
        assert gpu.counts()["refused"], name
        gpu.refuse("")
        t.run_steps(2)  # reported once
        t.close()


@pytest.mark.parametrize("form", [FP64, FP32])
def test_refused_launches_of_a_batch_are_reported(gpu, form):
    def grids():
        return [torch_b200.Torch(*blister(nx, ny), precision=form) for nx, ny in ((20, 33), (61, 17))]

    g = grids()
    b = torch_b200.Batch(g)
    b.run_steps(2, g[0].dt_max)  # the first steps are not captured
    gpu.reset()
    b.run_steps(6, g[0].dt_max)
    # (the column-density sweep has a graph of its own from the first steps, which takes over)
    names = [n for n in kernels(gpu) if "colden" not in n]
    assert gpu.counts()["graphs"] > 0
    b.close()
    for name in names:
        g = grids()
        b = torch_b200.Batch(g)
        b.run_steps(2, g[0].dt_max)
        gpu.reset()
        gpu.refuse(name)
        with pytest.raises(torch_b200.TrgError):
            b.run_steps(6, g[0].dt_max)
        assert gpu.counts()["refused"], name
        gpu.refuse("")
        b.close()


# ------------------------------------------------- shared memory of the chains
def strip(nx):
    """2-D, nx shells of at most 5 cells."""
    tp, ic = workloads.blister((nx, 3, 1), side=0.5 * workloads.PC2CM)
    return dataclasses.replace(tp, windCellRadius=0, massLossRate=0.0), ic


@pytest.mark.parametrize("form", [FP64, FP32])
@pytest.mark.parametrize("cells, chained", [(57000, True), (60000, False)])
def test_sweeps_of_very_many_shells_fit_a_cta_or_run_shell_by_shell(gpu, form, cells, chained):
    tp, ic = known_answers.spitzer_case(cells, 6.0) if form == FP64 else strip(cells)
    t = torch_b200.Torch(tp, ic, precision=form)
    t.run_steps(2)
    names = [l.name for l in gpu.launches()]
    t.close()
    assert gpu.counts()["refused"] == 0
    for sweep in ("rad", "colden"):
        assert any(f"k_{sweep}_chain" in n for n in names) == chained
        assert (sum(f"k_{sweep}_shell" in n for n in names) > cells - 20) == (not chained)


def test_batch_of_a_long_and_a_wide_grid_fits_a_cta(gpu):
    """The largest shell and the largest number of shells of different grids,
    taken together, ask for more than a CTA has; each grid asks for less."""
    wide = workloads.blister((500, 1000, 1))
    wide = dataclasses.replace(wide[0], windCellRadius=0, massLossRate=0.0), wide[1]
    grids = [torch_b200.Torch(*c) for c in (strip(50000), wide)]
    b = torch_b200.Batch(grids)
    gpu.reset()
    b.run_steps(3, grids[0].dt_max)
    chains = [l for l in gpu.launches() if "k_colden_chain" in l.name]
    b.close()
    assert gpu.counts()["refused"] == 0
    assert chains and all(l.grid == 2 and 48 * 1024 < l.smem <= 227 * 1024 for l in chains)


def test_kernel_attributes_do_not_depend_on_the_grid(gpu):
    """A kernel's shared-memory limit belongs to the device: set to one grid's
    need, it would fail another thread's larger grid between setting and launch."""
    for form in (FP64, FP32):
        grids = [torch_b200.Torch(*blister(nx, ny), precision=form) for nx, ny in ((300, 400), (20, 33))]
        for t in grids:
            t.run_steps(4)
        batch = [torch_b200.Torch(*blister(nx, ny), precision=form) for nx, ny in ((61, 17), (120, 90))]
        b = torch_b200.Batch(batch)
        b.run_steps(4, batch[0].dt_max)
        b.close()
    assert any("k_rad_chain" in l.name for l in gpu.launches())
    assert gpu.most_smem_settings() == 1


# ------------------------------------------------------- overlapped launches
@pytest.mark.parametrize("case", sorted(CASES))
def test_shell_overlap_switch_covers_every_launch(gpu, monkeypatch, case):
    """With TRG_SHELL_OVERLAP=0 no kernel may start while the one ahead of it
    runs; without, the step's kernels may."""
    make, form = CASES[case]
    tp, ic = make()
    for off in (False, True):
        if off:
            monkeypatch.setenv("TRG_SHELL_OVERLAP", "0")
        else:
            monkeypatch.delenv("TRG_SHELL_OVERLAP", raising=False)
        gpu.reset()
        t = torch_b200.Torch(tp, ic, precision=form)
        t.run_steps(6)
        if form == FP32:
            t.autotune()
        t.close()
        ahead = [l.name for l in gpu.launches() if l.programmatic]
        assert not ahead if off else len(ahead) > 6


# ------------------------------------------------------ restored checkpoints
@pytest.mark.parametrize("case, kept", [("hii_fp32", False), ("blister_fp64", False), ("sedov_fp32", True)])
def test_restored_time_step_minima_do_not_wait_for_a_kernel(gpu, case, kept):
    """A blob of a build that left the last step's minima in it: they are dt_max
    once the call has returned, with no kernel run after the copy (the hydro-only
    FP32 form's are the next step's limit and stay)."""
    make, form = CASES[case]
    t = torch_b200.Torch(*make(), precision=form)
    at = 8 + 2 * 4 + 8 + 4 * 4 + 8 + 4 * 4  # the header's scalars: dt, time, three minima, block count
    blob = bytearray(t.checkpoint())
    blob[at:at + 48] = struct.pack("6d", 0.25, 0.5, 1e-9, 2e-9, 3e-9, 7.0)
    t.restore(bytes(blob))
    got = struct.unpack("6d", t.checkpoint()[at:at + 48])
    want = (1e-9, 2e-9, 3e-9) if kept else (t.dt_max,) * 3
    t.close()
    assert got == (0.25, 0.5) + want + (0.0,)
