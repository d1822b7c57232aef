"""The work a user of mikroptim_b200 has it do, as cases that can be timed and checked.

Each case is one call (or one short chain of calls) through the package's public entry points:

  merit          engine.merit_device on an uploaded batch: the merit of every variant
  residuals      engine.residuals_device: residual rows, OPD and status of every ray
  run            engine.TraceEngine.run: host batch in, host residuals, OPD and status out
  gram           the fused adjoint + normal equations of run points (one variable set for all)
  gram_runs      the same for systems of uneven surface and variable counts
  gradient       autograd: the merit forward, its gradient backward
  jacobian       the materialised adjoint Jacobian and its normal equations
  jacobian_fd    the central-difference Jacobian and its normal equations
  lm             engine.optimize_lm_gpu: a batched Levenberg-Marquardt, host x0 in, x out
  eval           EVAL on the dense pupil grid: OPD maps, spots, field rays
  psf            scalar PSF and MTF of OPD maps

The systems are those of mikroptim_b200.workloads (singlets, seven-element objectives, uneven
element chains with a zero-power ghost plate, element chains of one length, toleranced
non-coaxial objectives), drawn anew from the seed. `exact` is a plain torch restatement in
float64 that shares no code with the package beyond the description of the systems.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from mikroptim_b200 import autograd as ag
from mikroptim_b200 import engine, psf, workloads
from mikroptim_b200.batch import (FAILURE_HARD, FAILURE_SOFT, PRECISION_FP64,
                                  PRECISION_FP64_FMA, PRECISION_MIXED, VAR_CURVATURE, VAR_GLASS,
                                  ResidualLayout)

DEVICE = "cuda"
PRECISION = {"fp64": PRECISION_FP64, "fp64_fma": PRECISION_FP64_FMA, "mixed": PRECISION_MIXED}


# ---- the cases -------------------------------------------------------------------------------
def listed():
    return [
        # an interactive edit of a lens: a handful of singlets, latency and launches count
        dict(name="merit_singlets", path="merit", system="singlet", variants=64,
             precision="fp64", soft=True),
        # one screening call from host arrays to host arrays, the size of configuration 1
        dict(name="run_singlets", path="run", system="singlet", variants=1024,
             precision="fp64", soft=True),
        # the dense-pupil sweep (20 surfaces, 9 wavelengths, 32 x 32 pupils), every row kept
        dict(name="residuals_sweep", path="residuals", system="sweep", variants=384,
             surfaces=20, wavelengths=9, rings=32, spokes=32, precision="fp64_fma", soft=True),
        # the merit of a multistart population of fast objectives (configuration 2)
        dict(name="merit_objectives", path="merit", system="objective", variants=4096,
             rings=16, spokes=32, glass=False, precision="fp64", soft=True),
        # the normal equations of such a population, curvatures, gaps and one glass variable
        dict(name="gram_objectives", path="gram", system="objective", variants=512,
             rings=16, spokes=32, glass=True, precision="fp64", soft=True),
        # systems of 6 to 30 surfaces and 8 to 56 variables in one call (configuration 3)
        dict(name="gram_uneven", path="gram_runs", system="uneven", variants=2048,
             rings=16, spokes=32, plate=True, precision="mixed", soft=True),
        # Monte-Carlo tolerancing: merit and gradient of decentered, tilted samples
        dict(name="gradient_tolerancing", path="gradient", system="tolerancing", variants=1024,
             elements=10, rings=16, spokes=32, precision="mixed", soft=True),
        # the Jacobian itself, as the default optimiser options and the diagnostics use it
        dict(name="jacobian_objectives", path="jacobian", system="objective", variants=48,
             rings=16, spokes=32, glass=False, exact_gram=True, precision="fp64", soft=True),
        # the reference method, finite differences, on many small systems
        dict(name="jacobian_fd_singlets", path="jacobian_fd", system="singlet", variants=1024,
             exact_gram=False, precision="fp64_fma", soft=True),
        # the optimiser end to end: upload, start, six iterations, results
        dict(name="lm_uneven", path="lm", system="uneven", variants=512, rings=16, spokes=32,
             plate=True, iterations=6, precision="fp64_fma", soft=True),
        # OPD maps and spots of finished designs
        dict(name="eval_objectives", path="eval", system="objective", variants=64, grid=64,
             half=False, precision="fp64", soft=True),
        # their PSF and MTF
        dict(name="psf_maps", path="psf", variants=32, grid=64, fft=256),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    path = rng.choice(["merit", "merit", "residuals", "run", "gram", "gram_runs", "gradient",
                       "jacobian", "jacobian_fd", "lm", "eval", "psf"])
    case = dict(path=path, precision="fp64", soft=rng.random() < 0.75)
    pupil = dict(rings=rng.randint(3, 20), spokes=rng.randint(4, 40))
    # variants of full-size pupils (16 x 32) worth of rays
    scale = max(1.0, 16.0 * 32.0 / (pupil["rings"] * pupil["spokes"]))
    if path in ("merit", "residuals"):
        system = rng.choice(["singlet", "objective", "sweep", "uneven"])
        case.update(system=system)
        if system == "singlet":
            case.update(variants=_log_int(rng, 1, 60000))
        elif system == "objective":
            case.update(pupil, variants=_log_int(rng, 1, 2000), glass=rng.random() < 0.3)
        elif system == "sweep":
            case.update(pupil, variants=_log_int(rng, 1, 500), surfaces=rng.randint(4, 24),
                        wavelengths=rng.randint(1, 9),
                        precision=rng.choice(["fp64", "fp64_fma"]))
        else:
            case.update(pupil, variants=_log_int(rng, 1, 800), plate=rng.random() < 0.7,
                        precision=rng.choice(["fp64", "fp64_fma"]))
    elif path == "run":
        case.update(system="singlet", variants=_log_int(rng, 1, 4000))
    elif path == "gram":
        system = rng.choice(["objective", "sweep", "singlet"])
        case.update(system=system)
        if system == "objective":
            case.update(pupil, variants=_log_int(rng, 1, int(300 * min(scale, 4))),
                        glass=rng.random() < 0.5)
        elif system == "sweep":
            case.update(pupil, variants=_log_int(rng, 1, int(300 * min(scale, 4))),
                        surfaces=rng.randint(4, 24), wavelengths=rng.randint(1, 9),
                        precision=rng.choice(["fp64", "fp64_fma", "mixed"]))
        else:
            case.update(variants=_log_int(rng, 1, 10000),
                        precision=rng.choice(["fp64", "fp64_fma", "mixed"]))
    elif path == "gram_runs":
        case.update(pupil, system="uneven", plate=rng.random() < 0.7,
                    variants=_log_int(rng, 1, int(500 * min(scale, 4))),
                    precision=rng.choice(["fp64", "fp64_fma", "mixed", "mixed"]))
    elif path == "gradient":
        case.update(pupil, system="tolerancing", elements=rng.randint(2, 12),
                    variants=_log_int(rng, 1, int(300 * min(scale, 4))),
                    precision=rng.choice(["fp64_fma", "mixed", "mixed"]))
    elif path in ("jacobian", "jacobian_fd"):
        system = rng.choice(["singlet", "objective", "sweep"])
        case.update(system=system, exact_gram=rng.random() < 0.5)
        if system == "singlet":
            case.update(variants=_log_int(rng, 1, 4000),
                        precision=rng.choice(["fp64", "fp64_fma"]))
        elif system == "objective":
            case.update(pupil, variants=_log_int(rng, 1, int(24 * min(scale, 4))), glass=False)
        else:
            case.update(pupil, variants=_log_int(rng, 1, int(24 * min(scale, 4))),
                        surfaces=rng.randint(4, 20), wavelengths=rng.randint(1, 7),
                        precision=rng.choice(["fp64", "fp64_fma"]))
    elif path == "lm":
        case.update(pupil, system="uneven", variants=_log_int(rng, 2, 300),
                    plate=rng.random() < 0.7, iterations=rng.randint(2, 6), soft=True,
                    precision="fp64_fma")
    elif path == "eval":
        case.update(system=rng.choice(["singlet", "objective"]), variants=_log_int(rng, 1, 48),
                    grid=rng.randint(9, 80), half=rng.random() < 0.4)
    else:
        grid = rng.randint(9, 96)
        case.update(grid=grid, fft=psf.psf_fft_size(grid, rng.choice([2.0, 4.0])),
                    variants=_log_int(rng, 1, 16))
    return case


# ---- inputs ----------------------------------------------------------------------------------
def _system(case, seed):
    """(batch, settings, variables, x0) of the case's systems."""
    failure = FAILURE_SOFT if case["soft"] else FAILURE_HARD
    common = dict(seed=20261203 + 1000003 * int(seed), failure=failure,
                  precision=PRECISION[case["precision"]])
    v, name = case["variants"], case["system"]
    if name == "singlet":
        return workloads.singlet(v, **common)
    common.update(rings=case.get("rings", 16), spokes=case.get("spokes", 32))
    if name == "objective":
        return workloads.objective(v, glass=case.get("glass", False), **common)
    if name == "sweep":
        return workloads.sweep(v, surfaces=case["surfaces"], wavelengths=case["wavelengths"],
                               **common)
    if name == "uneven":
        return _uneven(v, case["plate"], common)
    return workloads.tolerancing(v, elements=case["elements"], **common)


def _uneven(variants, plate, common):
    """Systems of uneven length, the first of them of the table's full length with all of its
    variables (so that the shapes of the results do not hang on the draw)."""
    out, full = (workloads.uneven(n, plate=plate, **extra, **common) for n, extra in (
        (variants, {}), (1, dict(s_min=30, s_max=30, p_min=64, p_max=64))))
    batch, settings, variables, x0 = out
    for name in ("curvature", "thickness", "index", "pupil_radius", "field_angle",
                 "field_target", "variant_surfaces"):
        getattr(batch, name)[0] = getattr(full[0], name)[0]
    variables[0], x0[0] = full[2][0], full[3][0]
    return batch, settings, variables, x0


WAVELENGTHS_PSF = workloads.OBJECTIVE_WAVELENGTHS
FIELDS_PSF = 5


def _maps(case, seed):
    """OPD maps [T][N][N] in mm: low-order aberrations of up to about a wave, NaN outside the
    pupil and, in every third map, in a vignetted segment; with their wavelengths in mm."""
    n = case["grid"]
    T = case["variants"] * FIELDS_PSF * len(WAVELENGTHS_PSF)
    rng = np.random.default_rng(77000 + int(seed))
    lam = np.tile(np.array(WAVELENGTHS_PSF) * 1e-6, T // len(WAVELENGTHS_PSF))
    c = torch.from_numpy(rng.normal(0.0, 0.25, (T, 8)) * lam[:, None]).to(DEVICE)
    cut = torch.from_numpy(np.where(np.arange(T) % 3 == 2, rng.uniform(0.5, 1.0, T), 2.0))
    a = (2.0 * torch.arange(n, dtype=torch.float64, device=DEVICE) + 1.0 - n) / n
    y, x = a[:, None].expand(n, n), a[None, :].expand(n, n)
    r2 = x * x + y * y
    basis = torch.stack([r2, r2 * r2, x * y, x * x - y * y, x * r2, y * r2, x, y])
    maps = torch.einsum("tk,kij->tij", c, basis)
    bad = (r2 > 1.0)[None] | (y[None] > cut.to(DEVICE)[:, None, None])
    maps[bad] = float("nan")
    return maps, lam


def prepare(case, seed):
    path = case["path"]
    if path == "psf":
        maps, lam = _maps(case, seed)
        n = case["grid"]
        k = 2 * np.arange(n) + 1 - n
        full = float(np.count_nonzero(k[:, None] ** 2 + k[None, :] ** 2 <= n * n))
        pupil = [psf._capi.PsfPupilParams(float(w), 1.0 / (full * full), 1, 1) for w in lam]
        return dict(case=case, maps=maps, pupil=pupil)
    batch, settings, variables, x0 = _system(case, seed)
    layout = ResidualLayout(batch.topology, settings)
    state = dict(case=case, batch=batch, settings=settings, layout=layout, variables=variables)
    if path == "run":
        state["engine"] = engine.TraceEngine(0)
        state["trace"] = engine.TraceSettings(settings, opd=True)
        state["out"] = engine.TraceOutput()  # a loop hands its result back for reuse
        return state
    if path == "lm":
        state["x0"] = x0
        state["options"] = engine.LmOptions(max_iterations=case["iterations"], gram_exact=False,
                                            fail_weight_factor=1.0)
        return state
    if path == "gradient":
        state["problem"] = ag.AdjointProblem(batch, layout, variables)
        state["x"] = torch.from_numpy(np.ascontiguousarray(x0)).to(DEVICE)
        return state
    state["device"] = engine.DeviceSystemBatch(batch)
    if path == "gram_runs":
        runs = engine.RunVariables(variables)
        state["variables"] = runs
        state["x"] = torch.from_numpy(engine.pad_rows(x0, runs.runs, runs.pmax)).to(DEVICE)
    elif path in ("gram", "jacobian", "jacobian_fd"):
        state["x"] = torch.from_numpy(np.ascontiguousarray(x0)).to(DEVICE)
    elif path == "eval":
        state["eval"] = engine.EvalSettings(grid=case["grid"], half_pupil=case["half"])
    return state


# ---- one pass --------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    path = case["path"]
    if path == "psf":
        return psf.psf_device(state["maps"], state["pupil"], case["grid"], case["fft"])
    batch, layout = state["batch"], state["layout"]
    if path == "merit":
        o = engine.merit_device(state["device"], layout, batch)
        return o.merit, o.failed, o.hard_failed
    if path == "residuals":
        o = engine.residuals_device(state["device"], layout, batch)
        return o.residuals, o.opd, o.status
    if path == "run":
        o = state["engine"].run(batch, engine.TraceMode.RESIDUALS, state["trace"],
                                state["out"]).residuals
        return o.residuals, o.opd, o.status
    if path == "gram":
        return engine.adjoint_normal_equations_device(state["device"], layout, batch,
                                                      state["variables"], state["x"])
    if path == "gram_runs":
        return engine.adjoint_normal_equations_runs_device(state["device"], layout, batch,
                                                           state["variables"], state["x"])
    if path == "gradient":
        x = state["x"].detach().requires_grad_(True)
        merit = ag.merit(x, state["problem"])
        merit.sum().backward()
        return merit.detach(), x.grad
    if path == "jacobian":
        J, r, status = engine.adjoint_jacobian_device(state["device"], layout, batch,
                                                      state["variables"], state["x"])
        return J, r, status, engine.normal_equations_device(J, r, exact=case["exact_gram"])
    if path == "jacobian_fd":
        J, r, changes = engine.fd_jacobian_device(state["device"], layout, batch,
                                                  state["variables"], state["x"])
        return J, r, changes, engine.normal_equations_device(J, r, exact=case["exact_gram"])
    if path == "lm":
        o = engine.optimize_lm_gpu(batch, layout, state["variables"], state["x0"],
                                   state["options"])
        return o["x"], o["merit"]
    _, _, _, o = engine.evaluate_device_tensors(state["device"], batch, state["eval"])
    return o["opd"], o["sx"], o["sy"], o["st"], o["fr"], o["fs"]


# ---- the work a pass cannot do without -------------------------------------------------------
_SHAPE = {  # surfaces, wavelengths, fields on the axis, other fields, variables
    "singlet": (3, 3, 1, 2, 4), "objective": (15, 7, 1, 4, 29)}


def _shape(case):
    """(mean surfaces, wavelengths x fields, rays, variables) of one variant."""
    name = case["system"]
    rings, spokes = case.get("rings", 16), case.get("spokes", 32)
    if name == "singlet":
        rings, spokes = 6, 12
    if name in _SHAPE:
        S, L, axis, other, P = _SHAPE[name]
        P += 3 if case.get("glass") else 0
    elif name == "sweep":
        S, L, axis, other = case["surfaces"], case["wavelengths"], 0, 5
        P = 1 + 3 * ((S - 1) // 2)
    elif name == "uneven":
        S, L, axis, other, P = 18, 7, 0, 5, 26
    else:
        S, L, axis, other = 1 + 2 * case["elements"], 7, 0, 5
        P = 4 * case["elements"]
    return S, L * (axis + other), L * (axis * rings + other * rings * spokes), P


def work(case):
    """Bytes read and written once, and floating-point operations by the reference's own cost
    model: 140 per ray and surface step (two more steps per ray for the start and the reference
    sphere), 3 times that for a forward and reverse sweep, 4 P per ray for the row, 2 P^2 per
    row for its normal equations; 5 N log2 N per transform of N complex values."""
    v, path = case["variants"], case["path"]
    if path == "psf":
        T, n, m = v * FIELDS_PSF * len(WAVELENGTHS_PSF), case["grid"], case["fft"]
        lines = 5.0 * m * math.log2(m)
        return {"bytes": T * 8.0 * (n * n + m * m + 2 * (n + 1)),
                "flops": T * (lines * (n + m) + 4.0 * m * m)}
    S, tuples, rays, P = _shape(case)
    record = 8.0 * (2 * S + S * 9 + 16)
    rows = rays * (2 if case["soft"] else 1)
    trace = 140.0 * (S + 1)
    if path == "merit":
        return {"bytes": v * (record + 24.0), "flops": v * rays * trace}
    if path in ("residuals", "run"):
        return {"bytes": v * (record + rows * 8.0 + rays * 9.0), "flops": v * rays * trace}
    if path in ("gram", "gram_runs", "gradient"):
        return {"bytes": v * (record + 8.0 * (P + 1) ** 2),
                "flops": v * rays * (3.0 * trace + 4.0 * P + 2.0 * P * P)}
    if path == "jacobian":
        return {"bytes": v * (record + rows * 8.0 * (P + 1) + rays),
                "flops": v * (rays * (3.0 * trace + 4.0 * P) + rows * 2.0 * P * P)}
    if path == "jacobian_fd":
        return {"bytes": v * (record + rows * 8.0 * (P + 1)),
                "flops": v * (rays * (2 * P + 1) * trace + rows * (3.0 * P + 2.0 * P * P))}
    if path == "lm":
        cycle = rays * (4.0 * trace + 4.0 * P + 2.0 * P * P)
        return {"bytes": v * (record + 16.0 * P), "flops": v * case["iterations"] * cycle}
    points = math.pi / 4.0 * case["grid"] ** 2 * (0.5 if case["half"] else 1.0)
    return {"bytes": v * (record + tuples * points * 25.0), "flops": v * tuples * points * trace}


# ---- how far another correct implementation may be off ---------------------------------------
def tolerance(case):
    """About four times what the path was seen to differ by from `exact`, or between its own
    precision modes; the FP64 mode's arithmetic is fixed operation by operation except for the
    order of the sums on the tensor cores."""
    path, precision = case["path"], case.get("precision", "fp64")
    fp64 = precision == "fp64"
    if path == "psf":
        return {"rel": 2e-15, "max": 2e-14}  # seen: 3.2e-16, 2.4e-15
    if path in ("merit", "residuals", "run", "eval") and fp64:
        return "exact"
    if path == "merit":
        return {"rel": 2e-11, "max": 2e-10}
    if path == "residuals":  # the OPD is what is left of path lengths 1e5 times as long
        return {"rel": 4e-10, "max": 4e-9}  # seen: 5.0e-11, 4.9e-10
    if path in ("gram", "gram_runs"):
        if precision == "mixed":
            return {"rel": 1e-6, "max": 1e-5}  # seen: 1.2e-7, 3.4e-7
        if case["system"] == "objective":
            # rays continued past a miss or a total reflection amplify a rounding by up to 1e11
            return {"rel": 1e-10, "max": 1e-8}
        return {"rel": 1e-13, "max": 1e-12}  # seen: 2.6e-15, 1.1e-14
    if path == "gradient":
        # seen: 2.7e-7, 1.3e-6 (FP32 reverse sweep) and 2.5e-13, 5.4e-13
        return {"rel": 1e-6, "max": 1e-5} if precision == "mixed" else {"rel": 2e-12, "max": 2e-11}
    if path in ("jacobian", "jacobian_fd") and fp64:
        return "exact" if case["exact_gram"] else {"rel": 1e-12, "max": 1e-10}
    if path == "jacobian":
        return {"rel": 1e-10, "max": 4e-10}  # seen: 1.4e-11, 5.0e-11
    if path == "jacobian_fd":  # differences of residuals over steps of 6e-6
        return {"rel": 1e-6, "max": 1e-5}  # seen: 2.3e-7, 1.9e-6
    # lm: nearly collinear thickness columns; FP64 with and without contraction ends this far
    # apart (an FP32 reverse sweep 3e-2: its trajectories cannot be compared)
    return {"rel": 1e-9, "max": 5e-8}  # seen: 2.0e-10, 1.2e-8


# ---- plain torch in float64 ------------------------------------------------------------------
OK, MISSED, TIR, BACKWARD, SOFT_MISSED, SOFT_TIR = 0, 1, 2, 3, 5, 6
EXACT_SECONDS_OF_RAY_STEPS = 1.5e10  # ray-surface steps of a reverse sweep in about 15 s


class _Pupil:
    """Field, wavelength, weight and pupil position of every ray of a variant, in row order."""

    def __init__(self, topo, rings, spokes):
        x, w = np.polynomial.legendre.leggauss(rings)
        rho, w = np.sqrt(0.5 * (x + 1.0)), 0.5 * w
        f, l, r, phi, wt = [], [], [], [], []
        for fi in range(topo.fields):
            mode = int(topo.pupil_mode[fi])  # 0 half, 1 full, 2 axis
            m = 1 if mode == 2 else spokes
            a = (2.0 * np.arange(m) + 1.0) * math.pi / (m * (2 if mode == 0 else 1))
            a = np.zeros(1) if mode == 2 else a
            for li in range(topo.wavelengths):
                f.append(np.full(rings * m, fi))
                l.append(np.full(rings * m, li))
                r.append(np.repeat(rho, m))
                phi.append(np.tile(a, rings))
                wt.append(np.repeat(w / m, m))
        put = lambda a: torch.from_numpy(np.concatenate(a)).to(DEVICE)
        self.f, self.l, self.weight = put(f), put(l), put(wt)
        rho, phi = put(r), put(phi)
        self.x, self.y = rho * torch.sin(phi), rho * torch.cos(phi)
        self.tuple = self.f * topo.wavelengths + self.l
        self.tuples = topo.fields * topo.wavelengths


class _Systems:
    """The parameters of variants [a, b) as float64 tensors."""

    def __init__(self, batch, a, b):
        put = lambda x: torch.from_numpy(np.ascontiguousarray(x[a:b])).to(DEVICE)
        self.S, self.L = batch.surfaces, batch.wavelengths
        self.sphere = [int(t) == 2 for t in batch.type]
        self.c, self.t, self.n = put(batch.curvature), put(batch.thickness), put(batch.index)
        self.pupil, self.target = put(batch.pupil_radius), put(batch.field_target)
        self.sin, self.cos = torch.sin(put(batch.field_angle)), torch.cos(put(batch.field_angle))
        self.xf = put(batch.decenter_tilt) if batch.decenter_tilt is not None else None
        self.count = (put(batch.variant_surfaces).long() if batch.variant_surfaces is not None
                      else torch.full((b - a,), self.S, dtype=torch.long, device=DEVICE))
        self.omega = None
        if batch.buchdahl_coeff is not None:
            self.buchdahl = put(batch.buchdahl_coeff)
            self.omega = torch.from_numpy(batch.buchdahl_omega()).to(DEVICE)

    def parameters(self, l):
        """Curvatures, thicknesses and indices as one tensor per surface ([V][1], and the
        index at every ray's wavelength [V][R]), ready to be replaced by expanded leaves."""
        c = [self.c[:, s:s + 1] if self.sphere[s] else None for s in range(self.S)]
        t = [self.t[:, s:s + 1] for s in range(self.S)]
        n = [self.n[:, s, :][:, l] for s in range(self.S)]
        return c, t, n

    def apply(self, variables, x):
        """The parameters with variables x [V][P] written into them."""
        self.c, self.t, self.n = self.c.clone(), self.t.clone(), self.n.clone()
        for k, var in enumerate(variables.variables):
            if var.type == VAR_CURVATURE:
                self.c[:, var.surface] = x[:, k]
            elif var.type == VAR_GLASS:
                self.buchdahl = self.buchdahl.clone()
                self.buchdahl[:, var.surface, var.component] = x[:, k]
            else:
                self.t[:, var.surface] = x[:, k]
        for s in {v.surface for v in variables.variables if v.type == VAR_GLASS}:
            b, w = self.buchdahl[:, s, :, None], self.omega[None, :]
            self.n[:, s] = b[:, 0] + w * (b[:, 1] + w * (b[:, 2] + w * b[:, 3]))


def _sqrt(x, ok):
    return torch.sqrt(torch.where(ok, x, torch.ones_like(x)))


def _div(a, b, ok):
    return a / torch.where(ok, b, torch.ones_like(b))


def _rotate(x, y, z, ca, sa, cb, sb):
    """R^T v of R = R_y(b) R_x(a)."""
    x, z = cb * x - sb * z, sb * x + cb * z
    return x, ca * y + sa * z, ca * z - sa * y


def _rotate_back(x, y, z, ca, sa, cb, sb):
    y, z = ca * y - sa * z, sa * y + ca * z
    return cb * x + sb * z, y, cb * z - sb * x


def _trace(sys, params, start, field, soft):
    """Rays through the surfaces: a dict of status, opl (up to the last surface), penalty,
    first soft event and the state. Every quantity is [V][R]."""
    c, t, n = params
    px, py = start
    zero, one = torch.zeros_like(px), torch.ones_like(px)
    dx, dy, dz = zero, sys.sin[:, field] + zero, sys.cos[:, field] + zero
    pz, opl, pen = zero, py * dy, zero
    status = torch.zeros_like(px, dtype=torch.long)
    first = torch.zeros_like(status)
    count = sys.count[:, None]
    for s in range(1, sys.S):
        live = (status == OK) & (s < count)
        back = live & ~(dz > 0)
        go = live & ~back
        status = torch.where(back, BACKWARD, status)
        pz1 = pz - t[s - 1]
        ox, oy, oz, ux, uy, uz = px, py, pz1, dx, dy, dz
        tilt = None
        if sys.xf is not None:
            q = sys.xf[:, s]
            tilt = [torch.cos(q[:, 2:3]), torch.sin(q[:, 2:3]), torch.cos(q[:, 3:4]),
                    torch.sin(q[:, 3:4])]
            ox, oy, oz = _rotate(ox - q[:, 0:1], oy - q[:, 1:2], oz, *tilt)
            ux, uy, uz = _rotate(ux, uy, uz, *tilt)
            back = go & ~(uz > 0)
            status = torch.where(back, BACKWARD, status)
            go = go & ~back
        s0 = _div(-oz, uz, go)
        x, y = ox + s0 * ux, oy + s0 * uy
        cs = c[s] if c[s] is not None else zero
        H = cs * (x * x + y * y)
        B = uz - cs * (x * ux + y * uy)
        D = B * B - cs * H
        miss = go & (D < 0)
        if not soft:
            status = torch.where(miss, MISSED, status)
            go, miss = go & ~miss, torch.zeros_like(miss)
        root = _sqrt(D, go & ~miss & (D > 0)) * ((D > 0) | miss)
        denom = B + root
        lost = go & ~miss & ~(denom > 0)
        status = torch.where(lost, MISSED, status)
        go = go & ~lost
        sl = torch.where(miss, _div(B, cs + zero, miss), _div(H, denom, go & ~miss))
        pen = torch.where(miss, pen - D, pen)
        first = torch.where(miss & (first == OK), SOFT_MISSED, first)
        x, y, z = x + sl * ux, y + sl * uy, sl * uz
        opl = torch.where(go, opl + n[s - 1] * (s0 + sl), opl)
        nx, ny, nz = -cs * x, -cs * y, one - cs * z
        inv = torch.where(miss, 1.0 / _sqrt(nx * nx + ny * ny + nz * nz, miss), one)
        nx, ny, nz = inv * nx, inv * ny, inv * nz
        mu = n[s - 1] / n[s]
        ci = ux * nx + uy * ny + uz * nz
        k = one - mu * mu * (one - ci * ci)
        tir = go & (k < 0)
        if not soft:
            status = torch.where(tir, TIR, status)
            go, tir = go & ~tir, torch.zeros_like(tir)
        pen = torch.where(tir, pen - k, pen)
        first = torch.where(tir & (first == OK), SOFT_TIR, first)
        a = _sqrt(k, go & ~tir & (k > 0)) * (k > 0) - mu * ci
        ex, ey, ez = ux - ci * nx, uy - ci * ny, uz - ci * nz
        inv = 1.0 / _sqrt(ex * ex + ey * ey + ez * ez, tir)
        ex, ey, ez = (torch.where(tir, inv * e, mu * u + a * m)
                      for e, u, m in ((ex, ux, nx), (ey, uy, ny), (ez, uz, nz)))
        if tilt is not None:
            x, y, z = _rotate_back(x, y, z, *tilt)
            x, y = x + q[:, 0:1], y + q[:, 1:2]
            ex, ey, ez = _rotate_back(ex, ey, ez, *tilt)
        px, py, pz = (torch.where(go, u, v) for u, v in ((x, px), (y, py), (z, pz)))
        dx, dy, dz = (torch.where(go, u, v) for u, v in ((ex, dx), (ey, dy), (ez, dz)))
    return dict(status=status, first=first, opl=opl, pen=pen, p=(px, py, pz), d=(dx, dy, dz))


def _last(sys, values):
    """Each variant's value at its own last surface."""
    if all(int(c) == sys.S for c in sys.count[:1]) and bool((sys.count == sys.S).all()):
        return values[-1] + torch.zeros_like(values[0] + values[-1])
    out = values[-1]
    for s in range(sys.S - 1):
        out = torch.where(sys.count[:, None] == s + 1, values[s], out)
    return out


def _to_sphere(sys, ray, params, field, soft):
    """The step onto the reference sphere through the last vertex: status, opl, penalty."""
    _, t, n = params
    (px, py, pz), (dx, dy, dz) = ray["p"], ray["d"]
    h, w, n_image = sys.target[:, field], _last(sys, t), _last(sys, n)
    status, first = ray["status"], ray["first"]
    status = torch.where((status == OK) & (first != OK), first, status)
    live = (status == OK) | (status == SOFT_MISSED) | (status == SOFT_TIR)
    back = live & ~(dz > 0)
    status = torch.where(back, BACKWARD, status)
    live = live & ~back
    b = -(px * dx + (py - h) * dy + (pz - w) * dz)
    g = px * px + py * (py - 2.0 * h) + pz * (pz - 2.0 * w)
    disc = b * b - g
    miss = live & (disc < 0)
    if not soft:
        status = torch.where(miss, MISSED, status)
        live, miss = live & ~miss, torch.zeros_like(miss)
    root = _sqrt(disc, live & ~miss & (disc > 0)) * (disc > 0)
    denom = torch.where(w >= 0, b + root, b - root)
    lost = live & ~miss & ~torch.where(w >= 0, denom > 0, denom < 0)
    status = torch.where(lost, MISSED, status)
    live = live & ~lost
    status = torch.where(miss & (status == OK), SOFT_MISSED, status)
    first = torch.where(miss & (first == OK), SOFT_MISSED, first)
    pen = torch.where(miss, ray["pen"] - _div(disc, h * h + w * w, miss), ray["pen"])
    step = torch.where(miss, b, _div(g, denom, live & ~miss))
    opl = torch.where(live, ray["opl"] + n_image * step, ray["opl"])
    return status, opl, pen, first, live


def _weights(batch, settings, pupil):
    """Residual and penalty scale of every ray's tuple times the root of its weight."""
    wf = np.asarray(batch.field_weight) / np.sum(batch.field_weight)
    wl = np.asarray(batch.wavelength_weight) / np.sum(batch.wavelength_weight)
    w = torch.from_numpy((wf[:, None] * wl[None, :]).reshape(-1)).to(DEVICE)[pupil.tuple]
    scale = torch.sqrt(w) / (batch.reference_wavelength_nm * 1e-6)
    root = torch.sqrt(pupil.weight)
    return scale * root, torch.sqrt(settings.fail_weight * w) * root


def _per_tuple(pupil, values):
    """Sums over the rays of each tuple [V][tuples]."""
    out = torch.zeros(values.shape[0], pupil.tuples, dtype=values.dtype, device=DEVICE)
    return out.index_add(1, pupil.tuple, values)


def _centre(pupil, live, values):
    """values less their weighted mean over the tuple's live rays; 0 for the others."""
    w = pupil.weight * live
    total = _per_tuple(pupil, w)
    mean = _per_tuple(pupil, w * torch.where(live, values, 0.0)) / torch.where(total > 0, total, 1.0)
    return torch.where(live, values - mean[:, pupil.tuple], 0.0)


def _rays(sys, params, pupil, soft):
    start = sys.pupil[:, None] * pupil.x, sys.pupil[:, None] * pupil.y
    ray = _trace(sys, params, start, pupil.f, soft)
    return _to_sphere(sys, ray, params, pupil.f, soft)


def _rows(batch, settings, pupil, sys, params):
    """Residual rows, penalty rows (or None), OPD and status."""
    soft = settings.failure == FAILURE_SOFT
    status, opl, pen, _, live = _rays(sys, params, pupil, soft)
    scale, pscale = _weights(batch, settings, pupil)
    opd = _centre(pupil, live, opl)
    fail = torch.where(status == OK, 0.0, torch.where(live, pen, pen + 1.0))
    return scale * opd, pscale * fail if soft else None, opd, status


def _chunks(batch, rays, most=600_000):
    step = max(1, most // max(rays, 1))
    return [(a, min(a + step, batch.variants)) for a in range(0, batch.variants, step)]


def _jacobian(batch, settings, pupil, sys, sets):
    """Rows [V][rows] and their derivatives [V][rows][P] by reverse mode: every ray gets its own
    copy of each parameter, so one sweep gives the derivatives of every ray."""
    soft = settings.failure == FAILURE_SOFT
    R, V = pupil.f.numel(), sys.c.shape[0]
    c, t, n = sys.parameters(pupil.l)
    leaf = {}
    for key in sorted({(0 if v.type == VAR_CURVATURE else 2 if v.type == VAR_GLASS else 1,
                        v.surface) for vs in sets for v in vs.variables}):
        lst = (c, t, n)[key[0]]
        lst[key[1]] = leaf[key] = (lst[key[1]].expand(V, R).clone()).requires_grad_(True)
    status, opl, pen, first, live = _rays(sys, (c, t, n), pupil, soft)
    scale, pscale = _weights(batch, settings, pupil)
    keys = list(leaf)

    def grads(value, mask):
        out = torch.autograd.grad((torch.where(mask, value, 0.0)).sum(), [leaf[k] for k in keys],
                                  retain_graph=True, allow_unused=True)
        return {k: torch.zeros(V, R, dtype=torch.float64, device=DEVICE) if g is None else g
                for k, g in zip(keys, out)}

    g_opl = grads(opl, live)
    g_pen = grads(pen, first != OK) if soft and pen.requires_grad else None
    P = max(vs.size for vs in sets)
    J = torch.zeros(V, R * (2 if soft else 1), P, dtype=torch.float64, device=DEVICE)

    def column(g, v, var):
        kind = 0 if var.type == VAR_CURVATURE else 2 if var.type == VAR_GLASS else 1
        out = g[(kind, var.surface)][v]
        return out * sys.omega[pupil.l] ** var.component if kind == 2 else out

    same = len(sets) == 1
    with torch.no_grad():
        for v in [slice(None)] if same else range(V):
            for k, var in enumerate(sets[0 if same else v].variables):
                J[v, :R, k] = column(g_opl, v, var)
                if g_pen is not None:
                    J[v, R:, k] = pscale * column(g_pen, v, var)
        for k in range(P):
            J[:, :R, k] = scale * _centre(pupil, live, J[:, :R, k])
        r = scale * _centre(pupil, live, opl)
        if soft:
            fail = torch.where(status == OK, 0.0, torch.where(live, pen, pen + 1.0))
            r = torch.cat([r, pscale * fail], dim=1)
    return r, J, status


def _exact_gram(case, batch, settings, variables, x0):
    pupil = _Pupil(batch.topology, settings.rings, settings.spokes)
    R = pupil.f.numel()
    many = isinstance(variables, list)
    pmax = max(v.size for v in variables) if many else variables.size
    out = torch.zeros(batch.variants, (pmax + 1) ** 2, dtype=torch.float64, device=DEVICE)
    for a, b in _chunks(batch, R):
        sys = _Systems(batch, a, b)
        if sys.omega is not None:
            sys.apply(variables, torch.from_numpy(np.ascontiguousarray(x0[a:b])).to(DEVICE))
        sets = variables[a:b] if many else [variables]
        r, J, _ = _jacobian(batch, settings, pupil, sys, sets)
        X = torch.cat([J, r[:, :, None]], dim=2)
        G = X.transpose(1, 2) @ X
        for v in range(b - a):
            P = sets[v].size if many else pmax
            keep = torch.tensor(list(range(P)) + [G.shape[1] - 1], device=DEVICE)
            out[a + v, :(P + 1) ** 2] = G[v][keep][:, keep].reshape(-1)
    return out.reshape(-1, pmax + 1, pmax + 1)


def _exact_gradient(batch, settings, variables, x0):
    pupil = _Pupil(batch.topology, settings.rings, settings.spokes)
    merits, grads = [], []
    for a, b in _chunks(batch, pupil.f.numel()):
        sys = _Systems(batch, a, b)
        x = torch.from_numpy(np.ascontiguousarray(x0[a:b])).to(DEVICE).requires_grad_(True)
        sys.apply(variables, x)
        r, p, _, _ = _rows(batch, settings, pupil, sys, sys.parameters(pupil.l))
        m = (r * r).sum(1) + ((p * p).sum(1) if p is not None else 0.0)
        m.sum().backward()
        merits.append(m.detach())
        grads.append(x.grad)
    return torch.cat(merits), torch.cat(grads)


def _exact_jacobian(batch, settings, variables, x0):
    pupil = _Pupil(batch.topology, settings.rings, settings.spokes)
    out = []
    for a, b in _chunks(batch, pupil.f.numel()):
        sys = _Systems(batch, a, b)
        r, J, status = _jacobian(batch, settings, pupil, sys, [variables])
        X = torch.cat([J, r[:, :, None]], dim=2)
        out.append((J.transpose(1, 2).contiguous(), r, status.to(torch.uint8),
                    X.transpose(1, 2) @ X))
    return tuple(torch.cat(o) for o in zip(*out))


def _exact_fd(batch, settings, variables, x0):
    """Central differences with the step 2^(-52/3) max(|x|, typical) about an interior point."""
    pupil = _Pupil(batch.topology, settings.rings, settings.spokes)
    x0 = torch.from_numpy(np.ascontiguousarray(x0)).to(DEVICE)
    typical = torch.from_numpy(variables.typical()).to(DEVICE)
    h = 2.0 ** (-52.0 / 3.0) * torch.maximum(x0.abs(), typical)
    lo, up = (torch.from_numpy(a).to(DEVICE) for a in (variables.lower(), variables.upper()))
    if bool(((x0 + h > up) | (x0 - h < lo)).any()):
        return None
    out = []
    for a, b in _chunks(batch, pupil.f.numel()):
        def rows(x):
            sys = _Systems(batch, a, b)
            sys.apply(variables, x)
            r, p, _, status = _rows(batch, settings, pupil, sys, sys.parameters(pupil.l))
            return (r if p is None else torch.cat([r, p], dim=1)), status == OK
        x = x0[a:b]
        r, ok = rows(x)
        J = torch.empty(b - a, variables.size, r.shape[1], dtype=torch.float64, device=DEVICE)
        changes = torch.empty(b - a, variables.size, dtype=torch.int64, device=DEVICE)
        for k in range(variables.size):
            xp, xm = x.clone(), x.clone()
            xp[:, k] += h[a:b, k]
            xm[:, k] -= h[a:b, k]
            (rp, okp), (rm, okm) = rows(xp), rows(xm)
            step = (xp[:, k] - x[:, k]) - (xm[:, k] - x[:, k])
            J[:, k] = (rp - rm) / step[:, None]
            changes[:, k] = ((okp != ok) | (okm != ok)).sum(1)
        X = torch.cat([J, r[:, None]], dim=1)
        out.append((J, r, changes, X @ X.transpose(1, 2)))
    return tuple(torch.cat(o) for o in zip(*out))


def _exact_rows(batch, settings, merit):
    pupil = _Pupil(batch.topology, settings.rings, settings.spokes)
    out = []
    for a, b in _chunks(batch, pupil.f.numel(), 4_000_000):
        sys = _Systems(batch, a, b)
        r, p, opd, status = _rows(batch, settings, pupil, sys, sys.parameters(pupil.l))
        if merit:
            m = (r * r).sum(1) + ((p * p).sum(1) if p is not None else 0.0)
            hard = (status != OK) & (status != SOFT_MISSED) & (status != SOFT_TIR)
            out.append((m, (status != OK).sum(1), hard.sum(1)))
        else:
            out.append((r if p is None else torch.cat([r, p], dim=1), opd,
                        status.to(torch.uint8)))
    return tuple(torch.cat(o) for o in zip(*out))


def _exact_eval(case, batch):
    """The dense grid: spots at the image plane, OPD at the sphere about the image point through
    the paraxial exit pupil, the field rays. Every failure is hard."""
    N, F, L = case["grid"], batch.fields, batch.wavelengths
    k = 2 * np.arange(N) + 1 - N
    inside = k[:, None] ** 2 + k[None, :] ** 2 <= N * N
    gx, gy = np.broadcast_to(k[None, :], (N, N)), np.broadcast_to(k[:, None], (N, N))
    keep = inside & (gx >= 0) if case["half"] else inside
    full = float(inside.sum())
    X, Y = gx[keep] / N, gy[keep] / N
    W = np.where(case["half"] & (gx[keep] > 0), 2.0, 1.0) / full
    n = X.size
    d = 1e-3
    X, Y = np.concatenate([X, [0.0, 0.0, 0.0, d]]), np.concatenate([Y, [0.0, d, -d, 0.0]])
    pts = torch.from_numpy(np.stack([X, Y])).to(DEVICE)
    W = torch.from_numpy(W).to(DEVICE)
    nan = float("nan")
    parts = []
    for a, b in _chunks(batch, F * L * n, 4_000_000):
        sys = _Systems(batch, a, b)
        V, T = b - a, F * L
        field = torch.arange(F, device=DEVICE).repeat_interleave(L * (n + 4))
        lam = torch.arange(L, device=DEVICE).repeat_interleave(n + 4).repeat(F)
        params = sys.parameters(lam)
        x, y = pts.repeat(1, T)
        ray = _trace(sys, params, (sys.pupil[:, None] * x, sys.pupil[:, None] * y), field, False)
        (px, py, pz), (dx, dy, dz) = ray["p"], ray["d"]
        status = torch.where((ray["status"] == OK) & ~(dz > 0), BACKWARD, ray["status"])
        ok = status == OK
        h, w = sys.target[:, field], sys.t[:, -1:]
        s0 = _div(w - pz, dz, ok)
        ix, iy = px + s0 * dx, py + s0 * dy
        # the paraxial chief ray (wavelength column 0): exit pupil -y / u' behind the last vertex
        yy, u, nb = torch.zeros_like(w), torch.ones_like(w), 1.0
        for s in range(sys.S):
            nn = sys.n[:, s, 0:1]
            if s > 0:
                yy = yy + sys.t[:, s - 1:s] * u
            u = (nb * u - yy * (sys.c[:, s:s + 1] * (nn - nb))) / nn
            nb = nn
        dz_ap = w + yy / u
        radius = torch.hypot(sys.target, dz_ap)
        kappa = (torch.sign(dz_ap) / radius)[:, field]
        qx, qy, qz = px, py - h, pz - w
        bq = -(qx * dx + qy * dy + qz * dz)
        t = -((qy * dz - qz * dy) ** 2 + (qz * dx - qx * dz) ** 2 + (qx * dy - qy * dx) ** 2)
        disc = 1.0 + kappa * kappa * t
        lost = ok & ~(disc >= 0)
        status = torch.where(lost, MISSED, status)
        ok = ok & ~lost
        step = bq - kappa * t / (_sqrt(disc, ok) + 1.0)
        opl = torch.where(ok, ray["opl"] + params[2][-1] * step, ray["opl"])
        shape = lambda q: q.reshape(V, T, n + 4)
        opl, ok, status, ix, iy, h = (shape(q) for q in (opl, ok, status, ix, iy, h + 0.0 * ix))
        dirs = [shape(q) for q in (dx, dy, dz)]
        chief = torch.where(ok[:, :, n:n + 1], opl[:, :, n:n + 1], 0.0)
        o, g = opl[:, :, :n] - chief, ok[:, :, :n]
        total = (W * g).sum(2, keepdim=True)
        piston = (W * torch.where(g, o, 0.0)).sum(2, keepdim=True) / total
        blank = lambda v, m: torch.where(m, v, nan)
        fo = ok[:, :, n:]
        fr = torch.stack([blank(v[:, :, n:], fo) for v in (ix, iy - h, *dirs)], dim=3)
        parts.append((blank(o - piston, g).reshape(-1), blank(ix[:, :, :n], g).reshape(-1),
                      blank((iy - h)[:, :, :n], g).reshape(-1),
                      status[:, :, :n].reshape(-1).to(torch.uint8), fr.reshape(-1),
                      status[:, :, n:].reshape(-1).to(torch.uint8)))
    return tuple(torch.cat(q) for q in zip(*parts))


def _exact_psf(case, seed):
    maps, lam = _maps(case, seed)
    n, m = case["grid"], case["fft"]
    k = 2 * np.arange(n) + 1 - n
    full = float(np.count_nonzero(k[:, None] ** 2 + k[None, :] ** 2 <= n * n))
    out, cuts = [], []
    for a in range(0, maps.shape[0], 256):
        part = maps[a:a + 256]
        w = torch.from_numpy(lam[a:a + 256]).to(DEVICE)[:, None, None]
        phase = 2.0 * math.pi * torch.nan_to_num(part / w)
        field = torch.where(torch.isnan(part), 0.0, torch.exp(1j * phase))
        intensity = torch.fft.fft2(field, s=(m, m)).abs() ** 2 / (full * full)
        otf = torch.fft.ifft2(intensity).abs()
        z = otf[:, :1, :1]
        cuts.append(torch.stack([otf[:, 0, :n + 1], otf[:, :n + 1, 0]], dim=1) / z)
        out.append(torch.fft.fftshift(intensity, dim=(1, 2)))
    return torch.cat(out), torch.cat(cuts)


def exact(case, seed):
    path = case["path"]
    if path == "lm":
        return None  # a reverse sweep in plain torch of every run and iteration takes minutes
    if path == "psf":
        return _exact_psf(case, seed)
    batch, settings, variables, x0 = _system(case, seed)
    S, _, rays, _ = _shape(case)
    if path in ("gram", "gram_runs", "gradient", "jacobian") and \
            float(case["variants"]) * rays * S > EXACT_SECONDS_OF_RAY_STEPS:
        return None
    if path in ("gram", "gram_runs"):
        return _exact_gram(case, batch, settings, variables, x0)
    if path == "gradient":
        return _exact_gradient(batch, settings, variables, x0)
    if path == "jacobian":
        return _exact_jacobian(batch, settings, variables, x0)
    if path == "jacobian_fd":
        return _exact_fd(batch, settings, variables, x0)
    if path == "eval":
        return _exact_eval(case, batch)
    return _exact_rows(batch, settings, path == "merit")
