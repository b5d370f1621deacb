"""Performance cases: what a program that runs this library has it do.

A host program sets a run up once (grid, star, tables, sweep order), then hands
the library a conserved state, lets it take K full steps (Torch::fullStep) and
takes the new state back - to write a snapshot, to couple another module, to
stop at a checkpoint.  One pass of a case is that: state in, K steps, state
out, through the Python class or, where the state is large, through the C ABI
with the program's own pinned buffers (what bench.py times end to end).  K is
a stretch between two snapshots, so that the steps and not the copies are the
bulk of a pass.

The cases cover the two precision forms (FP64, bit-exact with the reference;
FP32), hydrodynamics alone and with radiation and cooling, one, two and three
dimensions, cartesian, cylindrical and spherical grids, single grids and
batches, even and odd sizes, from a 1-D tube of a few hundred cells, where a
step is a handful of launches, to the 256^3 grids the library is benchmarked
on.
"""
import ctypes
import dataclasses
import math

import numpy as np
import torch

import torch_b200
from torch_b200 import config, setups, workloads

PC = workloads.PC2CM
FORMS = {"fp64": torch_b200.PRECISION_FP64, "fp32": torch_b200.PRECISION_FP32}


def listed():
    return [
        # A 1-D shock tube (the Sod problem the tests use as a known answer): the
        # smallest grids there are, where the launches of a step are its time.
        dict(name="sod_1d_fp64", kind="hydro", nx=400, ny=1, nz=1, form="fp64", riemann="HLLC", warm=2, steps=60),
        # A 1-D spherical HII region (the D-type expansion known answer): radiation
        # transfer along one ray, one cell per shell.
        dict(name="spitzer_1d_fp64", kind="spitzer", nx=200, form="fp64", warm=40, steps=12),
        # The shipped configuration: 150 x 200 cylindrical blister HII region with
        # stellar wind, radiation and cooling, in both forms.
        dict(name="blister_2d_fp64", kind="blister", nx=150, ny=200, form="fp64", warm=30, steps=12),
        dict(name="blister_2d_fp32", kind="blister", nx=150, ny=200, form="fp32", warm=30, steps=12),
        # A 2-D blast wave at an odd size in the FP64 form.
        dict(name="sedov_2d_fp64", kind="hydro", nx=257, ny=257, nz=1, form="fp64", riemann="RotatedHLLC", warm=10,
             steps=60),
        # 3-D Sedov blasts, hydrodynamics alone: the benchmark's 256^3 in the FP32
        # form, and an odd grid in the FP64 form.
        dict(name="sedov_256_fp32", kind="hydro", nx=256, ny=256, nz=256, form="fp32", riemann="RotatedHLLC", warm=10,
             steps=30),
        dict(name="sedov_97_fp64", kind="hydro", nx=97, ny=97, nz=97, form="fp64", riemann="RotatedHLLC", warm=10,
             steps=18),
        # 3-D HII regions in a lognormal cloud, radiation and cooling: the headline
        # benchmark's 256^3 in the FP32 form, a small ragged grid in the FP32 form,
        # and a production-sized one in the FP64 form.
        dict(name="hii_256_fp32", kind="hii", n=256, form="fp32", warm=6, steps=24),
        dict(name="hii_75_fp32", kind="hii", n=75, form="fp32", warm=12, steps=24),
        dict(name="hii_100_fp64", kind="hii", n=100, form="fp64", warm=12, steps=12),
        # A parameter study: many independent 2-D cylindrical HII regions of uneven
        # sizes advanced together.
        dict(name="batch_64_fp32", kind="batch", grids=64, study=2024, nx_min=64, nx_max=256, ny_min=64, ny_max=320,
             form="fp32", warm=12, steps=12),
        # An embedding program that keeps its state on the GPU and may not allocate:
        # the allocation-free FP32 hydro step on its own device buffers.
        dict(name="noalloc_64", kind="noalloc", nx=64, ny=64, nz=64, warm=0, steps=30),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed kinds, sizes spread over their ranges."""
    kind = rng.choice(["hydro1", "hydro2", "hydro3", "hydro3", "spitzer", "blister", "blister", "hii", "hii", "batch",
                       "noalloc"])
    form = rng.choice(["fp64", "fp32"])
    if kind == "hydro1":
        return dict(kind="hydro", nx=_log_int(rng, 100, 3200), ny=1, nz=1, form="fp64",
                    riemann=rng.choice(["HLLC", "HLL"]), warm=2, steps=60)
    if kind == "hydro2":
        nx = _log_int(rng, 48, 640)
        return dict(kind="hydro", nx=nx, ny=_log_int(rng, 48, 640), nz=1, form=form, riemann="RotatedHLLC", warm=10,
                    steps=30)
    if kind == "hydro3":
        top = 200 if form == "fp32" else 112
        nx, ny, nz = (_log_int(rng, 24, top) for _ in range(3))
        return dict(kind="hydro", nx=nx, ny=ny, nz=nz, form=form, riemann=rng.choice(["RotatedHLLC", "HLLC"]), warm=10,
                    steps=18)
    if kind == "spitzer":
        return dict(kind="spitzer", nx=_log_int(rng, 60, 1000), form="fp64", warm=40, steps=12)
    if kind == "blister":
        return dict(kind="blister", nx=_log_int(rng, 48, 300), ny=_log_int(rng, 64, 400), form=form, warm=30, steps=12)
    if kind == "hii":
        return dict(kind="hii", n=_log_int(rng, 24, 160 if form == "fp32" else 96), form=form, warm=12, steps=12)
    if kind == "batch":
        return dict(kind="batch", grids=_log_int(rng, 4, 64), study=rng.randrange(1 << 30), nx_min=48, nx_max=_log_int(rng, 64, 256),
                    ny_min=64, ny_max=_log_int(rng, 80, 320), form=form, warm=12, steps=12)
    nx, ny, nz = (_log_int(rng, 16, 63) for _ in range(3))
    return dict(kind="noalloc", nx=nx, ny=ny, nz=nz, warm=0, steps=30)


# ----------------------------------------------------------------- inputs
def _rng(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(shape, gen):
    return torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64)


def _hydro_input(case, seed):
    """A Sod tube (1-D) or a Sedov blast (2-D, 3-D: 1e51 erg in a 3-cell
    radius, one cell high in 2-D, at the centre of the tests' uniform medium),
    the medium stirred by a seeded 2 per cent; the blast energy varies with the
    seed by up to a factor of two."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    nd = 1 if ny == 1 else (2 if nz == 1 else 3)
    gen = _rng(seed)
    side = 2 * PC
    tp = workloads.sedov_parameters(n=nx, nd=nd, riemann=case.get("riemann", "RotatedHLLC"), side=side)
    tp = dataclasses.replace(tp, ncells=(nx, ny, nz), star_position=(nx // 2, ny // 2, nz // 2))
    dx = side / nx
    stir = torch.exp(0.02 * _randn((nz, ny, nx), gen))
    if nd == 1:
        tp = dataclasses.replace(tp, heatCapacityRatio=1.4)
        left = (torch.arange(nx, device="cuda") < nx // 2).reshape(1, 1, nx)
        den = torch.where(left, 1.0e-20, 0.125e-20) * stir
        pre = torch.where(left, 1.0e-10, 1.0e-11).to(torch.float64).expand_as(den)
    else:
        axes = [(torch.arange(n, device="cuda", dtype=torch.float64) + 0.5 - 0.5 * n) for n in (nz, ny, nx)]
        r2 = axes[2].reshape(1, 1, nx) ** 2 + axes[1].reshape(1, ny, 1) ** 2
        if nd == 3:
            r2 = r2 + axes[0].reshape(nz, 1, 1) ** 2
        inside = r2 <= 9.0
        energy = 1e51 * 2.0 ** (2.0 * float(torch.rand((), generator=gen, device="cuda")) - 1.0)
        heat = (tp.heatCapacityRatio - 1.0) * energy / (float(inside.sum()) * dx ** 3)
        den = 1e-20 * stir
        pre = torch.where(inside, heat, 0.0) + 1e-12
    den, pre = den.reshape(-1).cpu().numpy(), pre.reshape(-1).cpu().numpy()
    ic = config.make_initial_conditions((nx, ny, nz), dx, den, pre, np.zeros(den.size), np.zeros((3, den.size)))
    return tp, ic


def _hii_input(case, seed):
    """The benchmark's lognormal cloud (setups.lognormal_cloud: mean 1e3
    cm^-3, sigma_ln 0.5, k^-11/3 spectrum, 100 K), its field drawn on the GPU."""
    n = case["n"]
    side = 2 * PC
    k = torch.fft.fftfreq(n, device="cuda", dtype=torch.float64) * n
    kk = torch.sqrt(k.reshape(n, 1, 1) ** 2 + k.reshape(1, n, 1) ** 2 + k.reshape(1, 1, n) ** 2)
    kk[0, 0, 0] = 1.0
    amp = kk ** (-11.0 / 6.0)
    amp[0, 0, 0] = 0.0
    gen = _rng(seed)
    field = torch.fft.ifftn(torch.complex(_randn((n, n, n), gen), _randn((n, n, n), gen)) * amp).real
    field = torch.exp((field - field.mean()) / field.std() * 0.5)
    den = (field * (1e3 / field.mean())).reshape(-1) * setups.HYDROGEN_MASS
    pre = den * (setups.SPECIFIC_GAS_CONSTANT * 100.0)
    den, pre = den.cpu().numpy(), pre.cpu().numpy()
    ic = config.make_initial_conditions((n, n, n), side / n, den, pre, np.zeros(den.size), np.zeros((3, den.size)))
    return workloads.hii_region_parameters(n=n, side=side), ic


def _spitzer_input(case, seed):
    """The tests' 1-D spherical HII region (uniform 400 cm^-3 and 300 K, 1e49
    photons/s, TTI coupling between 300 K and 8000 K, 6 pc), stirred by 2 per
    cent."""
    nx, side = case["nx"], 6 * PC
    tp = workloads.hii_region_parameters(n=nx, side=side, photon_rate=1e49)
    tp = dataclasses.replace(tp, nd=1, ncells=(nx, 1, 1), geometry="spherical", cooling_on=False, rt_coupling="tti",
                             THI=300.0, THII=8000.0, star_position=(0, 0, 0), faceSnap=(True, False, False),
                             leftBC=("reflecting",) * 3, rightBC=("outflow",) * 3, tmax=1.0e15)
    den = 400.0 * setups.HYDROGEN_MASS * torch.exp(0.02 * _randn((nx,), _rng(seed))).cpu().numpy()
    pre = den * (setups.SPECIFIC_GAS_CONSTANT * 300.0)
    return tp, config.make_initial_conditions((nx, 1, 1), side / nx, den, pre, np.zeros(nx), np.zeros((3, nx)))


def _blister_input(case, seed):
    """The shipped 2-D cylindrical setup at the case's size, its density
    profile stirred by 2 per cent."""
    tp, ic = workloads.blister((case["nx"], case["ny"], 1))
    stir = torch.exp(0.02 * _randn((ic.den.size,), _rng(seed))).cpu().numpy()
    return tp, dataclasses.replace(ic, den=ic.den * stir)


def _batch_inputs(case, seed):
    """The batch benchmark's parameter study (`study` draws the grids' sizes,
    photon rates and cloud profiles), each cloud stirred by 2 per cent."""
    gen = _rng(seed)
    out = []
    for tp, ic in workloads.blister_batch(G=case["grids"], seed=case["study"], nx_range=(case["nx_min"], case["nx_max"]),
                                          ny_range=(case["ny_min"], case["ny_max"])):
        stir = torch.exp(0.02 * _randn((ic.den.size,), gen)).cpu().numpy()
        out.append((tp, dataclasses.replace(ic, den=ic.den * stir)))
    return out


# ------------------------------------------------------------------ states
class _Steps:
    """State in, K steps, state out on one grid, the whole state returned
    through the Python class."""

    def __init__(self, case, tp, ic):
        self.sim = torch_b200.Torch(tp, ic, precision=FORMS[case["form"]])
        self.steps = case["steps"]
        self.sim.run_steps(case["warm"])
        self.U = self.sim.state().U

    def run(self):
        self.sim.set_conserved(self.U)
        dts = self.sim.run_steps(self.steps)
        s = self.sim.state()
        out = {"U": s.U, "Q": s.Q, "dts": dts}
        if self.has_star:
            out.update(R=s.R, T=s.T)
        return out

    has_star = False


class _RadSteps(_Steps):
    has_star = True


class _PinnedSteps:
    """The same for a large grid: the conserved state in the program's own
    pinned buffers, through the C ABI."""

    def __init__(self, case, tp, ic):
        self.sim = torch_b200.Torch(tp, ic, precision=FORMS[case["form"]])
        self.steps = case["steps"]
        self.sim.run_steps(case["warm"])
        self.U = torch.empty((7, self.sim.N), dtype=torch.float64, pin_memory=True)
        self.out = torch.empty((7, self.sim.N), dtype=torch.float64, pin_memory=True)
        self._get(self.U)

    def _get(self, buf):
        s = self.sim
        s._check(s.lib.trg_get_state(s.ctx, ctypes.c_void_p(buf.data_ptr()), None, None, None, None))

    def run(self):
        s = self.sim
        s._check(s.lib.trg_set_conserved(s.ctx, ctypes.c_void_p(self.U.data_ptr())))
        dts = s.run_steps(self.steps)
        self._get(self.out)
        return {"U": self.out, "dts": dts}


class _BatchSteps:
    """Every grid's state in, K batch steps, every grid's state out."""

    def __init__(self, case, inputs):
        self.grids = [torch_b200.Torch(tp, ic, precision=FORMS[case["form"]]) for tp, ic in inputs]
        self.batch = torch_b200.Batch(self.grids)
        self.steps = case["steps"]
        self.dt_next = min(g.dt_max for g in self.grids)
        sizes = [7 * g.N for g in self.grids]
        self.at = np.concatenate([[0], np.cumsum(sizes)]).tolist()
        self.U = torch.empty(self.at[-1], dtype=torch.float64, pin_memory=True)
        self.out = torch.empty(self.at[-1], dtype=torch.float64, pin_memory=True)
        self.batch.run_steps(case["warm"], self.dt_next)
        for i in range(len(self.grids)):
            self.batch.get_conserved(i, self.U.data_ptr() + 8 * self.at[i])
        self.batch.synchronize()

    def run(self):
        b = self.batch
        for i in range(len(self.grids)):
            b.set_conserved(i, self.U.data_ptr() + 8 * self.at[i])
        b.enqueue_steps(self.steps, self.dt_next)
        for i in range(len(self.grids)):
            b.get_conserved(i, self.out.data_ptr() + 8 * self.at[i])
        b.synchronize()
        return {"U": self.out}


class _NoAllocSteps:
    """K allocation-free hydro steps between the program's device buffers,
    each with the time step the one before allows."""

    def __init__(self, case, tp, ic):
        self.sim = torch_b200.Torch(tp, ic, precision=torch_b200.PRECISION_FP32)
        self.steps = case["steps"]
        self.gamma, self.nd = tp.heatCapacityRatio, ic.nd
        self.U = torch.from_numpy(self.sim.state().U).cuda()
        self.out = torch.empty_like(self.U)
        self.dt = _first_dt(self.U, tp, ic)

    def run(self):
        s, dt = self.sim, ctypes.c_double(self.dt)
        src = self.U
        for _ in range(self.steps):
            s._check(s.lib.trg_hydro_step_fp32_noalloc(s.ctx, ctypes.c_void_p(src.data_ptr()),
                                                       ctypes.c_void_p(self.out.data_ptr()), dt, ctypes.byref(dt),
                                                       None))
            src = self.out
        return {"U": self.out}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "hydro":
        tp, ic = _hydro_input(case, seed)
        return (_PinnedSteps if case["nz"] > 1 else _Steps)(case, tp, ic)
    if kind == "hii":
        return _PinnedSteps(case, *_hii_input(case, seed))
    if kind == "spitzer":
        return _RadSteps(case, *_spitzer_input(case, seed))
    if kind == "blister":
        return _RadSteps(case, *_blister_input(case, seed))
    if kind == "batch":
        return _BatchSteps(case, _batch_inputs(case, seed))
    return _NoAllocSteps(case, *_hydro_input(case, seed))


def run(state):
    return state.run()


# -------------------------------------------------------------------- work
def work(case):
    """Per step the state is read and written once (U; with a star also the
    optical depths and column densities), and per component sub-step of the
    operator split the arithmetic of its stencil is done: about 600 operations
    per face flux with its reconstruction, 100 per cell for the update, 300 per
    cell for a radiation or thermal sub-step."""
    kind = case["kind"]
    if kind == "batch":
        cells = case["grids"] * (case["nx_min"] + case["nx_max"]) / 2 * (case["ny_min"] + case["ny_max"]) / 2
        nd = 2
    elif kind == "hii":
        cells, nd = case["n"] ** 3, 3
    else:
        cells = case["nx"] * case.get("ny", 1) * case.get("nz", 1)
        nd = 1 + (case.get("ny", 1) > 1) + (case.get("nz", 1) > 1)
    hydro = 600 * nd + 100
    if kind in ("hydro", "noalloc"):
        word = 4 if case.get("form") == "fp32" or kind == "noalloc" else 8
        return {"bytes": case["steps"] * cells * 2.0 * 7 * word, "flops": case["steps"] * cells * 2.0 * hydro}
    return {"bytes": case["steps"] * cells * 2.0 * (7 + 6 + 4) * 8,
            "flops": case["steps"] * cells * (1.7 * hydro + 3.3 * 300)}


# ------------------------------------------------------------------- exact
# Hydrodynamics in plain torch, 64 bits: the MUSCL / RK2 scheme of the
# reference's Hydrodynamics and Fluid classes with albada slopes, HLL, HLLC and
# the rotated HLLC-HLL solver, outflow boundaries, cartesian cells.  A field is
# [nz, ny, nx]; a state is the list [density, pressure, HII, ADV, vx, vy, vz].
GAS_CONSTANT_CGS = 8.314462e7


class _Code:
    """Code units (density, pressure and time scales) and the floors in them."""

    def __init__(self, tp, ic):
        self.rho, self.p, self.t = tp.dscale, tp.pscale, tp.tscale
        self.v = math.sqrt(self.p / self.rho)
        self.gamma, self.X, self.nd = tp.heatCapacityRatio, tp.massFractionH, ic.nd
        self.dx = ic.dx / (self.v * self.t)
        self.dt_max = tp.tmax / self.t / 10.0
        self.Rg = GAS_CONSTANT_CGS / self.v ** 2
        self.dfloor, self.tfloor = tp.dfloor / self.rho, tp.tfloor
        self.pfloor = 0.1 * self.Rg * self.dfloor * self.tfloor
        self.shape = tuple(reversed(ic.ncells))


def _conserved(q, c):
    ke = 0.5 * q[0] * (q[4] ** 2 + q[5] ** 2 + q[6] ** 2)
    return [q[0], q[1] / (c.gamma - 1.0) + ke, q[0] * q[2], q[0] * q[3], q[0] * q[4], q[0] * q[5], q[0] * q[6]]


def _primitive(u, c, floors):
    ke = 0.5 * (u[4] ** 2 + u[5] ** 2 + u[6] ** 2) / u[0]
    q = [u[0], (u[1] - ke) * (c.gamma - 1.0)] + [u[f] / u[0] for f in range(2, 7)]
    if floors:
        q[2], q[3] = q[2].clamp(0.0, 1.0), q[3].clamp(0.0, 1.0)
        q[0], q[1] = q[0].clamp(min=c.dfloor), q[1].clamp(min=c.pfloor)
        mu = c.X * (q[2] + 1.0) + (1.0 - c.X) * 0.25
        cold = c.tfloor * mu * c.Rg * u[0]
        q[1] = torch.where(q[1] / (mu * c.Rg * q[0]) < c.tfloor, cold, q[1])
    return q


def _fixed(u, c):
    q = _primitive(u, c, False)
    x, a, den = q[2].clamp(0.0, 1.0), q[3].clamp(0.0, 1.0), u[0].clamp(min=c.dfloor)
    pre = q[1].clamp(min=c.pfloor)
    cold = (c.X * (x + 1.0) + (1.0 - c.X) * 0.25) * c.Rg * den * c.tfloor
    return _conserved([den, torch.maximum(pre, cold), x, a, q[4], q[5], q[6]], c)


def _albada(a, b):
    ab = a * b
    on = ab > 1e-30
    return torch.where(on, ab * (a + b) / torch.where(on, a * a + b * b, 1.0), 0.0)


def _along(q, n, c):
    """Physical flux of q along the unit normal n, and the speed along it."""
    un = q[4] * n[0] + q[5] * n[1] + q[6] * n[2]
    m = q[0] * un
    energy = q[1] * (c.gamma / (c.gamma - 1.0)) + 0.5 * q[0] * (q[4] ** 2 + q[5] ** 2 + q[6] ** 2)
    return un, [m, energy * un, m * q[2], m * q[3]] + [m * q[4 + k] + q[1] * n[k] for k in range(3)]


def _speeds(left, right, ul, ur, c):
    sl, sr = left[0].sqrt(), right[0].sqrt()
    s = sl + sr
    mean = (sl * ul + sr * ur) / s
    d2 = (sl * c.gamma * left[1] / left[0] + sr * c.gamma * right[1] / right[0]) / s
    d = (d2 + 0.5 * sr * sl / s ** 2 * (ur - ul) ** 2).sqrt()
    return mean - d, mean + d


def _hll(left, right, n, c):
    ul, fl = _along(left, n, c)
    ur, fr = _along(right, n, c)
    s_l, s_r = _speeds(left, right, ul, ur, c)
    cl, cr = _conserved(left, c), _conserved(right, c)
    out = []
    for f in range(7):
        mid = (s_r * fl[f] - s_l * fr[f] + s_l * s_r * (cr[f] - cl[f])) / (s_r - s_l)
        out.append(torch.where(s_r <= 0, fr[f], torch.where(s_l >= 0, fl[f], mid)))
    return out


def _hllc(left, right, n, c):
    ul, fl = _along(left, n, c)
    ur, fr = _along(right, n, c)
    s_l, s_r = _speeds(left, right, ul, ur, c)
    ml, mr = left[0] * (s_l - ul), right[0] * (s_r - ur)
    s_c = (right[1] - left[1] + ml * ul - mr * ur) / (ml - mr)
    on_left = s_c >= 0
    k = [torch.where(on_left, a, b) for a, b in zip(left, right)]
    fk = [torch.where(on_left, a, b) for a, b in zip(fl, fr)]
    s_k, u_k = torch.where(on_left, s_l, s_r), torch.where(on_left, ul, ur)
    uk = _conserved(k, c)
    m = k[0] * (s_k - u_k)
    a = m / (s_k - s_c)
    star = [a, a * (uk[1] / k[0] + (s_c - u_k) * (s_c + k[1] / m)), a * k[2], a * k[3]]
    star += [a * (k[4 + i] + (s_c - u_k) * n[i]) for i in range(3)]
    out = []
    for f in range(7):
        mid = fk[f] + s_k * (star[f] - uk[f])
        out.append(torch.where(s_l >= 0, fl[f], torch.where(s_r <= 0, fr[f], mid)))
    return out


def _face_flux(left, right, dim, c, riemann):
    d = [1.0 if k == dim else 0.0 for k in range(3)]
    if riemann == "HLL":
        return _hll(left, right, d, c)
    if riemann == "HLLC":
        return _hllc(left, right, d, c)
    # Rotated HLLC-HLL (Nishikawa & Kitamura 2008): HLL along the velocity
    # jump, HLLC across it; pure HLLC for no jump along the face normal, pure
    # HLL for no jump across it.
    dv = [right[4 + k] - left[4 + k] for k in range(3)]
    par = dv[dim]
    perp = [0.0 * par if k == dim else dv[k] for k in range(3)]
    pp = perp[0] ** 2 + perp[1] ** 2 + perp[2] ** 2
    r, s = (par ** 2 + pp).sqrt(), pp.sqrt()
    only_hllc = (r < 1e-6) | (par == 0)
    only_hll = ~only_hllc & (pp == 0)
    pure = only_hllc | only_hll
    r, s = torch.where(pure, 1.0, r), torch.where(pure, 1.0, s)
    sign = torch.where(par < 0, -1.0, 1.0)
    n1 = [torch.where(pure, d[k], sign * dv[k] / r) for k in range(3)]
    n2 = [torch.where(pure, d[k], s / r * d[k] - par / (r * s) * perp[k]) for k in range(3)]
    w1 = torch.where(only_hllc, 0.0, torch.where(only_hll, 1.0, par.abs() / r))
    w2 = torch.where(only_hllc, 1.0, torch.where(only_hll, 0.0, s / r))
    return [w1 * a + w2 * b for a, b in zip(_hll(left, right, n1, c), _hllc(left, right, n2, c))]


def _rates(q, c, riemann):
    """Flux divergence of the primitives q."""
    out = [torch.zeros_like(q[0]) for _ in range(7)]
    for dim in range(c.nd):
        axis = 2 - dim
        n = c.shape[axis]
        index = torch.arange(-2, n + 2, device="cuda").clamp(0, n - 1)
        wide = [x.index_select(axis, index) for x in q]
        low, high = wide[4 + dim].narrow(axis, 0, 2), wide[4 + dim].narrow(axis, n + 2, 2)
        low.copy_(torch.where(low > 0, -low, low))
        high.copy_(torch.where(high < 0, -high, high))
        left, right = [], []
        for x in wide:
            step = x.narrow(axis, 1, n + 3) - x.narrow(axis, 0, n + 3)
            half = 0.5 * _albada(step.narrow(axis, 0, n + 2), step.narrow(axis, 1, n + 2))
            mid = x.narrow(axis, 1, n + 2)
            left.append((mid + half).narrow(axis, 0, n + 1))
            right.append((mid - half).narrow(axis, 1, n + 1))
        flux = _face_flux(left, right, dim, c, riemann)
        for f in range(7):
            out[f] += (flux[f].narrow(axis, 0, n) - flux[f].narrow(axis, 1, n)) / c.dx
    return out


def _cfl(q, c):
    sound = (c.gamma * q[1] / q[0]).sqrt()
    rate = sum((q[4 + k].abs() + sound) / c.dx for k in range(c.nd))
    return 0.5 / float(rate.max())


def _hydro_step(u, dt, c, riemann):
    k1 = _rates(_primitive(u, c, True), c, riemann)
    half = _fixed([a + 0.5 * dt * b for a, b in zip(u, k1)], c)
    k2 = _rates(_primitive(half, c, False), c, riemann)
    return _fixed([a + dt * b for a, b in zip(u, k2)], c)


def _initial(ic, c):
    def field(x, unit):
        return torch.from_numpy(np.ascontiguousarray(x)).cuda().reshape(c.shape) / unit
    q = [field(ic.den, c.rho), field(ic.pre, c.p), field(ic.hii, 1.0), torch.zeros(c.shape, device="cuda", dtype=torch.float64)]
    return _conserved(q + [field(ic.vel[k], c.v) for k in range(3)], c)


def _first_dt(U, tp, ic):
    c = _Code(tp, ic)
    return min(_cfl(_primitive([x.reshape(c.shape) for x in U], c, True), c), c.dt_max)


def exact(case, seed):
    """Hydrodynamics in 64 bits; None with radiation and cooling, whose causal
    sweeps visit the cells shell after shell (minutes in plain torch)."""
    if case["kind"] not in ("hydro", "noalloc"):
        return None
    tp, ic = _hydro_input(case, seed)
    c, riemann = _Code(tp, ic), case.get("riemann", "RotatedHLLC")
    u, dts = _initial(ic, c), []
    if case["kind"] == "hydro":  # a run's first step is a tiny one
        dts.append(1e-20 * c.dt_max)
        u = _hydro_step(u, dts[0], c, riemann)
    while len(dts) < case["warm"] + case["steps"]:
        dts.append(min(_cfl(_primitive(u, c, True), c), c.dt_max))
        u = _hydro_step(u, dts[-1], c, riemann)

    def whole(x):
        return torch.stack([f.reshape(-1) for f in x])
    out = {"U": whole(u)}
    if case["kind"] == "hydro":
        out["dts"] = np.array(dts[case["warm"]:])
        if case["nz"] == 1:
            # the library's Q: the FP64 form leaves the predictor's primitives
            # of the last step, the FP32 form derives them from the new state
            out["Q"] = None
    return out
