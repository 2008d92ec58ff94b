"""The workloads whose speed is measured: what a program built on this package
spends its time in, through the package's public calls.

Six kinds of call, over the range of sizes the configurations use:

- `fields`: real fields expanded and synthesised on a SurfaceGrid (loads, sea
  levels, surface outputs).
- `spin`: spin-weighted batches, both directions (the strain tensor's parts).
- `sea_level`: the generalised sea-level equation's fixed point.
- `pass`: one pass of the within-step iteration through an open step.
- `maps`: the grid coupling's maps over every memory node.
- `run`, `ocean`, `adjoint`, `ensemble`: whole evolutions, as the headline
  benchmark, the coupled run, the sensitivity run and the calibration
  ensemble make them.

Inputs are synthetic and made from the seed: log-viscosity fields, caps and
land masks of `sl3dpp_gb300.configs`, coefficients decaying with the degree.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from sl3dpp_gb300 import configs
from sl3dpp_gb300.ensemble import Ensemble, elements_for
from sl3dpp_gb300.grid import SurfaceGrid
from sl3dpp_gb300.sealevel import SeaLevelSolver
from sl3dpp_gb300.viscoelastic3d import Evolution3D, Options, Viscoelastic3D, standard_earth

DEVICE = "cuda"
RTOL = 1e-10
# the mixed form's options, as the headline benchmark sets them
MIXED = dict(precision=1, correction_rtol=3e-6, correction_memory=10, warm_start=1, fp64_emulation=1)
# a body for the sea-level equation alone, non-dimensional
BODY = dict(omega=0.06, polar_moment=0.8, equatorial_moment=0.75, gravitational_constant=0.3, hc=-0.2, kc=0.15,
            m_u=0.3, m_phi=0.2, m_c=0.4)


def listed():
    return [
        # one surface load on the sea-level grid of a small run: the smallest call, bound by its launches
        {"name": "one_field_lmax32", "kind": "fields", "lmax": 32, "count": 1, "oversampling": 1.0, "emulation": False},
        # the spin -2 strain component of the second configuration's lateral nodes, in the default FP64 form
        {"name": "spin_fp64_lmax128", "kind": "spin", "lmax": 128, "N": -2, "count": 45, "emulation": False},
        # the same of the headline configuration's 55 lateral nodes, as its FP64 passes transform them
        {"name": "spin_emulated_lmax256", "kind": "spin", "lmax": 256, "N": -1, "count": 55, "emulation": True},
        # the sea-level equation under a growing ice load with axial rotation, the second configuration's grid
        {"name": "sea_level_lmax128", "kind": "sea_level", "lmax": 128, "rotation": 1},
        # one pass of a small odd-sized operator: an ordinary driver's iteration, latency and launches
        {"name": "pass_lmax45", "kind": "pass", "lmax": 45, "elements": 43, "ngll": 5, "kelvin": 0.0,
         "emulation": False},
        # one pass of the second configuration's operator (Burgers), the default FP64 form
        {"name": "pass_lmax128", "kind": "pass", "lmax": 128, "elements": 80, "ngll": 6, "kelvin": 0.5,
         "emulation": False},
        # the grid coupling's maps over all memory nodes
        {"name": "maps_lmax64", "kind": "maps", "lmax": 64, "elements": 53, "ngll": 5, "kelvin": 0.0,
         "emulation": False},
        # the first configuration: lmax 32, Maxwell, FP64; the start and four steps
        {"name": "run_fp64_lmax32", "kind": "run", "lmax": 32, "elements": 40, "ngll": 5, "kelvin": 0.0, "rms": 0.5,
         "mixed": False, "steps": 4, "scheme": "sdirk2"},
        # the headline benchmark's operator and options: the start and two steps of the mixed form
        {"name": "run_mixed_lmax256", "kind": "run", "lmax": 256, "elements": 120, "ngll": 6, "kelvin": 0.0,
         "rms": 1.0, "mixed": True, "steps": 2, "scheme": "sdirk2"},
        # the second configuration coupled to its ocean, mixed form: the start and two steps
        {"name": "ocean_mixed_lmax128", "kind": "ocean", "lmax": 128, "elements": 80, "ngll": 6, "kelvin": 0.5,
         "rms": 1.0, "mixed": True, "steps": 2},
        # the discrete adjoint of a short run: the backward direction
        {"name": "adjoint_lmax48", "kind": "adjoint", "lmax": 48, "elements": 45, "ngll": 5, "kelvin": 0.0,
         "rms": 0.5, "mixed": False, "steps": 2},
        # six members of the calibration ensemble at once, two steps each
        {"name": "ensemble_6", "kind": "ensemble", "members": 6, "lmax": 64, "steps": 2},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["fields", "spin", "spin", "sea_level", "pass", "pass", "maps", "run", "run", "ocean", "adjoint",
                       "ensemble"])
    if kind == "fields":
        return {"kind": kind, "lmax": log(12, 256), "count": log(1, 40), "oversampling": rng.choice([1.0, 1.5]),
                "emulation": False}
    if kind == "spin":
        return {"kind": kind, "lmax": log(24, 256), "N": rng.choice([-2, -1]), "count": log(3, 80),
                "emulation": rng.random() < 0.5}
    if kind == "sea_level":
        return {"kind": kind, "lmax": log(24, 256), "rotation": rng.choice([0, 1])}
    if kind in ("pass", "maps"):
        lmax = log(16, 144 if kind == "pass" else 96)
        return {"kind": kind, "lmax": lmax, "elements": rng.randint(max(24, elements_for(lmax) - 8),
                                                                    elements_for(lmax) + 4),
                "ngll": rng.choice([5, 6]), "kelvin": rng.choice([0.0, 0.5]), "emulation": rng.random() < 0.3}
    lmax = log(16, {"run": 128, "ocean": 96, "adjoint": 56, "ensemble": 80}[kind])
    if kind == "ensemble":
        return {"kind": kind, "members": rng.randint(3, 8), "lmax": lmax, "steps": rng.randint(1, 3)}
    mixed = rng.random() < 0.5 or lmax > 80
    case = {"kind": kind, "lmax": lmax, "elements": rng.randint(max(24, elements_for(lmax) - 8),
                                                                elements_for(lmax) + 4),
            "ngll": rng.choice([5, 6]), "kelvin": rng.choice([0.0, 0.5]), "rms": round(rng.uniform(0.3, 1.0), 3),
            "mixed": mixed, "steps": rng.randint(1, 2 if kind == "adjoint" else 3)}
    if kind == "run":
        case["scheme"] = rng.choice(["sdirk2", "backward_euler"])
    return case


# -- inputs ---------------------------------------------------------------------------------


def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed))


def _degrees(lmax):
    return torch.cat([torch.full((l + 1,), l) for l in range(lmax + 1)]).to(DEVICE)


def _real_coefficients(lmax, count, seed):
    """count fields' (l, m >= 0) coefficients, decaying as 1 / (l + 1)."""
    l = _degrees(lmax)
    c = torch.randn(count, l.numel(), dtype=torch.complex128, device=DEVICE, generator=_generator(seed))
    zonal = torch.tensor([k * (k + 1) // 2 for k in range(lmax + 1)], device=DEVICE)
    c[:, zonal] = c[:, zonal].real.to(torch.complex128)
    return (c / (l + 1.0)).reshape(-1)


def _spin_coefficients(lmax, N, count, seed):
    l = torch.cat([torch.full((2 * l + 1,), l) for l in range(abs(N), lmax + 1)]).to(DEVICE)
    c = torch.randn(count, l.numel(), dtype=torch.complex128, device=DEVICE, generator=_generator(seed))
    return (c / (l + 1.0)).reshape(-1)


def _field_size(lmax, oversampling):
    band = math.ceil(oversampling * lmax - 1e-12)
    nphi = 2 * band + 1
    while True:
        r = nphi
        for p in (2, 3, 5):
            while r % p == 0:
                r //= p
        if r == 1:
            return band + 1, nphi
        nphi += 1


def _sea_level_inputs(lmax, seed):
    """An ocean over an oblique basin, an ice load on the land and smooth Love
    numbers, on the lmax grid (numpy)."""
    rng = np.random.default_rng(seed)
    nt, nphi = _field_size(lmax, 1.0)
    theta = np.arccos(np.polynomial.legendre.leggauss(nt)[0][::-1])
    tt, pp = np.meshgrid(theta, 2 * np.pi * np.arange(nphi) / nphi, indexing="ij")
    a, b, lon = rng.uniform(0.3, 0.5), rng.uniform(0.1, 0.3), rng.uniform(0.0, 2.0 * np.pi)
    ocean = (np.cos(tt) < a + b * np.sin(2 * pp + lon)).astype(np.float64)
    ice = -0.5 * np.exp(-(((tt - rng.uniform(0.2, 0.4)) / 0.2) ** 2)) * (1.0 + 0.3 * np.cos(pp + lon)) * (1.0 - ocean)
    l = np.arange(lmax + 1.0)
    on = (l > 0).astype(np.float64)
    return dict(ocean=ocean, load=ice, h=-1.2 / (l + 1.0) * on, k=-0.5 / (l + 1.0) * on, l=0.3 / (l + 1.0) * on,
                ht=0.6 / (l + 1.0) * (l > 1), kt=0.3 / (l + 1.0) * (l > 1), lt=0.1 / (l + 1.0) * (l > 1))


def _operator(case, seed, **options):
    """An operator of the case with its delta field set: a seeded pattern to
    degree lmax / 4 between 100 and 670 km depth."""
    lmax = case["lmax"]
    opts = Options.defaults(lmax, case["ngll"], rtol=RTOL, max_iterations=120, **options)
    op = Viscoelastic3D(standard_earth(case["elements"], case["kelvin"], 10.0), opts)
    grid = SurfaceGrid(lmax, 0, opts.oversampling)
    c = configs.delta_coefficients(lmax, max(2, lmax // 4), case.get("rms", 1.0), seed)
    pattern = grid.SynthesiseBatch(torch.tensor(c, device=DEVICE), 1)
    depth = torch.tensor(configs.delta_indicator(op.radius), device=DEVICE)
    op.set_delta((depth[:, None] * pattern[None, :]).contiguous().view(-1))
    return op


def _cap(op, seed):
    """A polar cap of 2 km on the sea-level grid, non-dimensional: the field
    and its coefficients."""
    grid = SurfaceGrid(op.lmax, 0, 1.0)
    alpha = np.random.default_rng(seed).uniform(8.0, 18.0)
    cap = configs.cap_field(grid.theta, grid.nphi, alpha, 2000.0) / op.surface_density_scale
    return cap, grid.ExpandBatch(torch.tensor(cap, device=DEVICE), 1).cpu().numpy()


def _times(op, steps, years=500.0):
    return np.arange(steps + 1) * (years * configs.SECONDS_PER_YEAR / op.time_scale)


def _ramp(full, steps):
    return np.stack([full * (k + 1) / 10.0 for k in range(steps + 1)])


def prepare(case, seed):
    kind, lmax = case["kind"], case["lmax"]
    if kind == "fields":
        grid = SurfaceGrid(lmax, 0, case["oversampling"], fp64_emulation=case["emulation"])
        g = _generator(seed + 1)
        fields = torch.randn(case["count"] * grid.FieldSize(), dtype=torch.float64, device=DEVICE, generator=g)
        return dict(case=case, grid=grid, coefficients=_real_coefficients(lmax, case["count"], seed), fields=fields)
    if kind == "spin":
        grid = SurfaceGrid(lmax, 2, 1.5, fp64_emulation=case["emulation"])
        g = _generator(seed + 1)
        fields = torch.randn(case["count"] * grid.FieldSize(), dtype=torch.complex128, device=DEVICE, generator=g)
        return dict(case=case, grid=grid, coefficients=_spin_coefficients(lmax, case["N"], case["count"], seed),
                    fields=fields)
    if kind == "sea_level":
        p = _sea_level_inputs(lmax, seed)
        grid = SurfaceGrid(lmax, 0, 1.0)
        solver = SeaLevelSolver(grid, p["h"], p["k"], p["l"], p["ht"], p["kt"], p["lt"], rotation=case["rotation"],
                                **BODY)
        return dict(case=case, solver=solver, ocean=torch.tensor(p["ocean"].ravel(), device=DEVICE),
                    load=torch.tensor(p["load"].ravel(), device=DEVICE))
    if kind in ("pass", "maps"):
        op = _operator(case, seed, fp64_emulation=int(case["emulation"]))
        state = dict(case=case, op=op)
        if kind == "pass":
            # an open step of 500 yr under the cap, from rest, as a driver holds it
            _, full = _cap(op, seed)
            state["load"] = full
            state["memory"] = op.ZeroState()
            state["step"] = op.StartStep(state["memory"], _times(op, 1)[1], "backward_euler", 0.5 * full)
            state["strain"] = state["step"].StartStrain()
        else:
            n = op.layout()["spectral"]
            x = torch.randn(n, dtype=torch.complex128, device=DEVICE, generator=_generator(seed))
            # a real part's zonal coefficients are real
            P, L = op.node_count, lmax
            spin0 = ((L + 1) ** 2 - 4 + (L + 1) ** 2 - 1) * P
            x[spin0:spin0 + (L + 1) * P] = x[spin0:spin0 + (L + 1) * P].real.to(torch.complex128)
            state["strain"] = x
        return state
    if kind == "ensemble":
        rng = np.random.default_rng(seed)
        members = []
        for i in range(case["members"]):
            # sizes spread below the largest, the same for every seed
            m = max(8, int(round(lmax * (1.0 - 0.5 * i / case["members"]))))
            members.append({"lmax": m, "elements": elements_for(m), "ngll": 5, "rms": float(rng.uniform(0.3, 1.2)),
                            "ldelta": max(2, m // 4), "cap_degrees": float(rng.uniform(5.0, 20.0)),
                            "delta_seed": int(seed) * 100 + i, "steps": case["steps"]})
        return dict(case=case, ensemble=Ensemble(members, max_iterations=120))
    mixed = dict(MIXED) if case["mixed"] else {}
    op = _operator(case, seed, **mixed)
    cap, full = _cap(op, seed)
    steps = case["steps"]
    if kind == "ocean":
        grid = SurfaceGrid(lmax, 0, 1.0)
        land = grid.SynthesiseBatch(torch.tensor(configs.land_field_coefficients(lmax, seed), device=DEVICE), 1)
        op.set_ocean(configs.ocean_from_field(land.cpu().numpy(), grid.weights, grid.nphi, 0.3), rotation=1, rtol=RTOL)
        return dict(case=case, run=Evolution3D(op), times=_times(op, steps, 250.0), loads=_ramp(cap, steps))
    state = dict(case=case, run=Evolution3D(op, case.get("scheme", "sdirk2")), times=_times(op, steps),
                 loads=_ramp(full, steps))
    if kind == "adjoint":
        state["dual"] = _real_coefficients(lmax, steps + 1, seed).view(steps + 1, -1).cpu().numpy()
    return state


# -- the calls ------------------------------------------------------------------------------


class _StateStrain:
    """A state's strain coefficients where they are, on the device."""

    def __init__(self, state):
        self.state = state
        address, count = state.device_coefficients()
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<f8", "data": (address, False), "version": 3}


def _snapshots(out, names):
    got = {n: out[n] for n in names}
    got["strain"] = torch.as_tensor(_StateStrain(out["state"]), device=DEVICE)
    return got


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "fields":
        g, n = state["grid"], case["count"]
        return {"coefficients": g.ExpandBatch(state["fields"], n), "fields": g.SynthesiseBatch(state["coefficients"], n)}
    if kind == "spin":
        g, n, N = state["grid"], case["count"], case["N"]
        return {"coefficients": g.ExpandSpinBatch(N, state["fields"], n),
                "fields": g.SynthesiseSpinBatch(N, state["coefficients"], n)}
    if kind == "sea_level":
        out = state["solver"].solve_generalised(state["ocean"], rtol=1e-11, direct_load=state["load"])
        return {k: out[k] for k in ("sea_level_change", "displacement", "potential", "tangential_potential",
                                    "uniform_shift")} | {"angular_velocity": list(out["angular_velocity"])}
    if kind == "pass":
        step = state["step"]
        step.Respond(state["strain"])
        step.AddChannels(state["load"])
        after = step.StrainOf()
        return {"strain": after, "change": step.RelativeChange(after, state["strain"])}
    if kind == "maps":
        op = state["op"]
        c0, c1, r = op.SynthesiseTensor(state["strain"])
        back = op.AnalyseTensor(c0, c1, r)
        sph, tor = op.DegreeForces(back)
        return {"grid": [c0, c1, r], "spectral": back, "forces": [sph, tor], "strain": op.StrainOfSolutions(sph, tor)}
    if kind == "ensemble":
        out = state["ensemble"].run()
        return {"U": out["U"], "phi": out["phi"]}
    if kind == "ocean":
        return _snapshots(state["run"].RunOcean(state["times"], state["loads"]), ("U", "phi", "sea_level", "omega"))
    if kind == "adjoint":
        out = state["run"].Adjoint(state["times"], state["loads"], state["dual"], state["dual"])
        return {k: out[k] for k in ("objective", "load_kernels", "tide_kernels", "delta_gradient")}
    return _snapshots(state["run"].Run(state["times"], state["loads"]), ("U", "phi"))


# -- what the calls cannot do without -----------------------------------------------------


def _transform(lmax, N, real, oversampling, count):
    """(bytes, flops) of one transform of count fields, either direction: the
    coefficients and the fields once each; the Legendre contraction and the
    longitude transforms."""
    nt, nphi = _field_size(lmax, oversampling)
    rows = (lmax + 1) * (lmax + 2) // 2 if real else (lmax + 1) ** 2 - N * N
    coefficients, fields = 16.0 * rows * count, (8.0 if real else 16.0) * nt * nphi * count
    legendre = 2.0 * nt * rows * 2 * count
    rings = (2.5 if real else 5.0) * nphi * math.log2(nphi) * nt * count
    return coefficients + fields, legendre + rings


def _nodes(case, lateral):
    """About how many memory nodes an operator has (of an element's GLL points
    ngll - 1 are Gauss points; the lateral ones lie in 570 of the mantle's
    2891 km, the elements evenly over the solid radius)."""
    every = int(round(0.55 * case["elements"] * (case["ngll"] - 1)))
    return max(case["ngll"] - 1, every // 5) if lateral else every


def _pass(case, lateral=True):
    """(bytes, flops) of one pass of the within-step iteration: the iterate
    read and written, the lateral weight read; both transforms of the three
    tensor parts, and a band solve of every degree."""
    lmax, P = case["lmax"], _nodes(case, lateral)
    flops = 0.0
    for N, real in ((-2, False), (-1, False), (0, True)):
        flops += 2 * _transform(lmax, N, real, 1.5, P)[1]
    kd, dofs = 3 * case["ngll"], 2.5 * case["elements"] * (case["ngll"] - 1)
    flops += 2 * (lmax + 1) * (lmax + 2) / 2 * 4.0 * kd * dofs
    nt, nphi = _field_size(lmax, 1.5)
    return 2 * 16.0 * 2.5 * (lmax + 1) ** 2 * P + 8.0 * nt * nphi * P, flops


def work(case):
    kind, lmax = case["kind"], case["lmax"]
    if kind == "fields":
        b, f = _transform(lmax, 0, True, case["oversampling"], case["count"])
        return {"bytes": 2 * b, "flops": 2 * f}
    if kind == "spin":
        b, f = _transform(lmax, case["N"], False, 1.5, case["count"])
        return {"bytes": 2 * b, "flops": 2 * f}
    if kind == "sea_level":  # about a dozen iterations of both transforms; the inputs and outputs once
        _, f = _transform(lmax, 0, True, 1.0, 1)
        nt, nphi = _field_size(lmax, 1.0)
        return {"bytes": 8.0 * 6 * nt * nphi, "flops": 24 * f}
    if kind == "pass":
        b, f = _pass(case)
        return {"bytes": b, "flops": f}
    if kind == "maps":
        b = f = 0.0
        P = _nodes(case, False)
        for N, real in ((-2, False), (-1, False), (0, True)):
            x, y = _transform(lmax, N, real, 1.5, P)
            b, f = b + 2 * x, f + 2 * y
        return {"bytes": b, "flops": f}
    if kind == "ensemble":
        b = f = 0.0
        for i in range(case["members"]):
            m = max(8, int(round(lmax * (1.0 - 0.5 * i / case["members"]))))
            x, y = _pass({"lmax": m, "elements": elements_for(m), "ngll": 5})
            b, f = b + x, f + 60 * case["steps"] * y
        return {"bytes": b, "flops": f}
    # about thirty passes a stage whatever the form, two stages a step (the adjoint: forward and back);
    # the delta field and the strain once (the adjoint: its gradient too)
    stages = (1 + 2 * case["steps"]) * (2 if kind == "adjoint" else 1)
    _, f = _pass(case)
    nt, nphi = _field_size(lmax, 1.5)
    P = _nodes(case, False)
    b = P * (16.0 * 2.5 * (lmax + 1) ** 2 + (16.0 if kind == "adjoint" else 8.0) * nt * nphi)
    return {"bytes": b, "flops": 30 * stages * f}


# -- the exact results ------------------------------------------------------------------


def _lambda(lmax, N, m, x):
    """sqrt((2 l + 1) / 4 pi) d^l_{m N}(theta) for l = max(|m|, |N|) .. lmax
    over cos theta = x, N <= 0: the closed form at the lowest degree, then
    the three-term recurrence."""
    c, s = torch.sqrt((1.0 + x) / 2.0), torch.sqrt((1.0 - x) / 2.0)
    A, M = -N, abs(m)
    l0 = max(M, A)
    if M >= A:
        low, high = (s, c) if m >= 0 else (c, s)
        scale = 0.5 * (math.lgamma(2 * M + 1) - math.lgamma(M + A + 1) - math.lgamma(M - A + 1))
        d = torch.exp(scale + (M + A) * torch.log(low) + (M - A) * torch.log(high))
        sign = -1.0 if m >= 0 and (M + A) % 2 else 1.0
    else:
        scale = 0.5 * (math.lgamma(2 * A + 1) - math.lgamma(A + m + 1) - math.lgamma(A - m + 1))
        d = torch.exp(scale + (A - m) * torch.log(c) + (A + m) * torch.log(s))
        sign = -1.0 if (A + m) % 2 else 1.0
    rows, before, now = [], torch.zeros_like(x), sign * d
    for l in range(l0, lmax + 1):
        rows.append(math.sqrt((2 * l + 1) / (4 * math.pi)) * now)
        if l == 0:
            before, now = now, x.clone()
            continue
        up = (l + 1) * (2 * l + 1) / math.sqrt(((l + 1) ** 2 - m * m) * ((l + 1) ** 2 - N * N))
        down = math.sqrt((l * l - m * m) * (l * l - N * N)) / (l * (2 * l + 1))
        before, now = now, up * ((x - m * N / (l * (l + 1))) * now - down * before)
    return torch.stack(rows)


class _Transforms:
    """The plain transforms: a dense sum over the degrees at each order and a
    library FFT, float64."""

    def __init__(self, lmax, N, real, oversampling):
        self.lmax, self.N, self.real = lmax, N, real
        self.nt, self.nphi = _field_size(lmax, oversampling)
        x, w = np.polynomial.legendre.leggauss(self.nt)
        self.x = torch.tensor(x[::-1].copy(), device=DEVICE)
        self.w = torch.tensor(w[::-1].copy(), device=DEVICE)
        self.orders = range(0 if real else -lmax, lmax + 1)
        self.tables = {m: _lambda(lmax, N, m, self.x) for m in self.orders}

    def _at(self, m):
        ls = torch.arange(max(abs(m), abs(self.N)), self.lmax + 1, device=DEVICE)
        return ls * (ls + 1) // 2 + m if self.real else ls * ls - self.N * self.N + m + ls

    def synthesise(self, c, count):
        c = c.view(count, -1)
        h = torch.zeros(count, self.nt, self.nphi, dtype=torch.complex128, device=DEVICE)
        for m, t in self.tables.items():
            part = c[:, self._at(m)] @ t.to(torch.complex128)
            h[:, :, m % self.nphi] = part
            if self.real and m > 0:
                h[:, :, self.nphi - m] = part.conj()
        f = torch.fft.ifft(h, dim=2) * self.nphi
        return (f.real.contiguous() if self.real else f).reshape(-1)

    def expand(self, f, count):
        g = torch.fft.fft(f.view(count, self.nt, self.nphi).to(torch.complex128), dim=2)
        g = g * (2 * math.pi / self.nphi * self.w)[None, :, None]
        rows = (self.lmax + 1) * (self.lmax + 2) // 2 if self.real else (self.lmax + 1) ** 2 - self.N ** 2
        c = torch.zeros(count, rows, dtype=torch.complex128, device=DEVICE)
        for m, t in self.tables.items():
            c[:, self._at(m)] = g[:, :, m % self.nphi] @ t.T.to(torch.complex128)
        return c.reshape(-1)


def _exact_sea_level(case, seed):
    lmax = case["lmax"]
    p = {k: torch.tensor(v, device=DEVICE) for k, v in _sea_level_inputs(lmax, seed).items()}
    t = _Transforms(lmax, 0, True, 1.0)
    l = _degrees(lmax)
    ocean, load = p["ocean"], p["load"]

    def integral(f):
        return float((t.w * f.view(t.nt, t.nphi).sum(dim=1)).sum() * 2 * math.pi / t.nphi)

    area = integral(ocean)
    eustatic = -integral(load) / area
    factor = -(p["h"] + p["k"])  # gravity, density and radius one
    w, polar, G = BODY["omega"], BODY["polar_moment"], BODY["gravitational_constant"]
    axial_rotation, uniform = math.sqrt(16 * math.pi / 45) * w, -math.sqrt(16 * math.pi / 9) * w
    inertia, trace = math.sqrt(5 / (9 * math.pi)) * w / (G * polar), (4 / 3) * w / polar
    shell = (2 / 3) * w * math.sqrt(4 * math.pi) / polar
    h2, k2, ht2, kt2, lt2 = (float(p[n][2]) for n in ("h", "k", "ht", "kt", "lt"))
    denominator = 1 + inertia * kt2 * axial_rotation + trace * BODY["m_c"] * uniform

    def rotate(c):
        c20, c00 = float(c[3].real), float(c[0].real)
        omega = (-inertia * k2 * c20 - trace * (BODY["m_u"] + BODY["m_phi"]) * c00 - shell * c00) / denominator
        return omega, h2 * c20 + ht2 * axial_rotation * omega, k2 * c20 + kt2 * axial_rotation * omega

    def sea_level(c):
        s = factor[l] * c
        if case["rotation"]:
            omega, d20, g20 = rotate(c)
            s[3] = -(d20 + g20 + axial_rotation * omega)
            s[0] -= (BODY["hc"] + BODY["kc"] + 1) * uniform * omega
        field = t.synthesise(s, 1).view_as(ocean)
        shift = eustatic - integral(ocean * field) / area
        return field + shift, shift

    c = t.expand(load + ocean * eustatic, 1)
    # the fixed point with a least-squares history, to the rounding
    xs, fs = [], []
    for _ in range(60):
        field, shift = sea_level(c)
        g = t.expand(load + ocean * field, 1)
        f = torch.view_as_real(g - c).reshape(-1)
        xs, fs = xs[-6:] + [g], fs[-6:] + [f]
        if float(f.norm()) < 1e-15 * float(torch.view_as_real(c).norm()):
            break
        c = g
        if len(fs) > 1:
            d = torch.stack([fs[i + 1] - fs[i] for i in range(len(fs) - 1)], dim=1)
            gamma = torch.linalg.lstsq(d.cpu(), fs[-1].cpu()[:, None], driver="gelsd").solution[:, 0]
            for i, v in enumerate(gamma.tolist()):
                c = c - v * (xs[i + 1] - xs[i])
    field, shift = sea_level(c)
    d, pot, tan = p["h"][l] * c, p["k"][l] * c, p["l"][l] * c
    omega = 0.0
    if case["rotation"]:
        omega, d[3], pot[3] = rotate(c)
        d[0] += BODY["hc"] * uniform * omega
        pot[0] += BODY["kc"] * uniform * omega
        tan[3] += lt2 * axial_rotation * omega
    return {"sea_level_change": field.reshape(-1), "displacement": t.synthesise(d, 1),
            "potential": t.synthesise(pot, 1), "tangential_potential": t.synthesise(tan, 1), "uniform_shift": shift,
            "angular_velocity": [None, None, omega]}


def exact(case, seed):
    """The transforms and the sea-level equation in plain float64. A pass and
    what is built on passes would need the whole Earth model again: None."""
    kind = case["kind"]
    if kind == "sea_level":
        return _exact_sea_level(case, seed)
    if kind not in ("fields", "spin"):
        return None
    real = kind == "fields"
    N = 0 if real else case["N"]
    t = _Transforms(case["lmax"], N, real, case["oversampling"] if real else 1.5)
    n, g = case["count"], _generator(seed + 1)
    fields = torch.randn(n * t.nt * t.nphi, dtype=torch.float64 if real else torch.complex128, device=DEVICE,
                         generator=g)
    c = _real_coefficients(case["lmax"], n, seed) if real else _spin_coefficients(case["lmax"], N, n, seed)
    return {"coefficients": t.expand(fields, n), "fields": t.synthesise(c, n)}
