"""Timed cases of the solver: what a program built on this framework calls, over the sizes it calls it at.

Every case is a dict with a "kind" (one public path) and its sizes:

  hydro     a save interval of the resident hydro loop: state in, `steps` calls of rhllc.Hllc3dStab, state out
  con2prim  rhllc.GetPhysValueStab on a batch of conservative states
  scatter   illum.CalculateIntScattering + CalculateAllParam, FP64 in the reference's rounding order
  tc        illum.ScatterTC: scattering integral + moments on the tensor cores
  sweep     illum.CalculateIllum: one transport sweep over all directions
  coupled   rad_rhd.RadRHDStep: coupled radiation-hydro steps, state in and state out
  compton   illum.FullSpectrumScattering over the 100-bin spectrum
  ray       ray_tracing.RayTracer: one frame's intersections and its image

Meshes are the Kuhn meshes, directions the Fibonacci sets and inputs the distributions of the benchmark and the
tests.  `exact` restates each path in 64-bit torch without this package's kernels.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from radrhd_solver_b200 import _lib as L
from radrhd_solver_b200 import illum, rad_rhd, rhllc
from radrhd_solver_b200 import mesh as meshes
from radrhd_solver_b200 import ray_tracing as rt
from radrhd_solver_b200.c2p_mlp import LearnedGuess

DEV = "cuda:0"
CFL = 0.3
GAMMA_TUBE, GAMMA_JET = 5.0 / 3.0, 4.0 / 3.0
JET_INFLOW = (0.01, 0.0, 0.0, math.sqrt(1.0 - 1.0 / 49.0), 1e-3)  # rho, v (Lorentz factor 7 along +z), p
JET_EMISSION = (1.0, 10.0, math.pi, 1.0)
SPEEDS = (0.0, 1e-6, 1e-5, 0.3, 0.9, 0.99)  # gas speeds of the Compton cases, in units of c


def listed():
    return [
        # The plain-hydro configuration: a relativistic shock tube of 120,000 tetrahedra, where a step is a
        # launch and a read-back of the step's scalars.
        {"name": "hydro_tube_200x10x10", "kind": "hydro", "problem": "tube", "nx": 200, "ny": 10, "nz": 10,
         "steps": 20},
        # A jet production run between two saves, 1.57M cells.
        {"name": "hydro_jet_64", "kind": "hydro", "problem": "jet", "nx": 64, "ny": 64, "nz": 64, "steps": 10},
        # Primitive recovery of a whole snapshot (post-processing, restarts): 4M states, Lorentz factors to 50.
        {"name": "con2prim_4m", "kind": "con2prim", "n": 4_000_000},
        # The radiation half alone in reference rounding: 48^3 hexes, 256 directions, one group.
        {"name": "scatter_fp64_663k_256", "kind": "scatter", "rows": 663_552, "M": 256},
        # The same contraction where single precision is enough.
        {"name": "tc_f16x3_663k_256", "kind": "tc", "form": "f16x3", "rows": 663_552, "M": 256, "spread": False},
        # Many frequency groups over a fine direction set, values over 12 decades.
        {"name": "tc_f16x3_1m_512", "kind": "tc", "form": "f16x3", "rows": 1_048_576, "M": 512, "spread": True},
        # A small grey sweep: a few cells per direction and front, a test problem or a coarse level.
        {"name": "sweep_fp64_12_64", "kind": "sweep", "n": 12, "M": 64, "G": 1, "precision": "fp64",
         "item_geometry": False},
        # A production grey sweep on the 48^3 mesh.
        {"name": "sweep_fp64_48_256", "kind": "sweep", "n": 48, "M": 256, "G": 1, "precision": "fp64",
         "item_geometry": False},
        # Coupled jet, plain FP64 form: the reference's arithmetic throughout.
        {"name": "coupled_plain_32", "kind": "coupled", "n": 32, "M": 256, "G": 4, "form": "plain", "steps": 2},
        # Coupled jet, mixed-precision sweep, tensor-core scattering and the learned pressure guess.
        {"name": "coupled_chosen_48", "kind": "coupled", "n": 48, "M": 256, "G": 4, "form": "chosen", "steps": 2},
        # Frequency-coupled Compton scattering of two cells per SM.
        {"name": "compton_296_256", "kind": "compton", "cells": 296, "M": 256},
        # One frame of a light curve: 600 x 300 rays against 44,032 triangles.
        {"name": "ray_frame_48_64", "kind": "ray", "n_box": 48, "n_sphere": 64, "mode": rt.SURFACE, "frame": 11},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: sizes log-uniform over each path's range, odd and ragged ones among them."""
    kind = rng.choice(["hydro", "con2prim", "scatter", "tc", "sweep", "sweep", "coupled", "compton", "ray"])
    if kind == "hydro":
        if rng.random() < 0.5:
            n = _log_int(rng, 20, 300)
            return {"kind": kind, "problem": "tube", "nx": n, "ny": rng.randint(2, 12), "nz": rng.randint(2, 12),
                    "steps": rng.randint(5, 20)}
        n = _log_int(rng, 12, 60)
        return {"kind": kind, "problem": "jet", "nx": n, "ny": n, "nz": n, "steps": rng.randint(3, 10)}
    if kind == "con2prim":
        return {"kind": kind, "n": _log_int(rng, 1000, 4_000_000)}
    if kind == "scatter":
        return {"kind": kind, "rows": _log_int(rng, 500, 400_000), "M": rng.choice([26, 64, 100, 128, 195, 256])}
    if kind == "tc":
        return {"kind": kind, "form": rng.choice(["f16x3", "f16x3", "bf16x3", "f16"]),
                "rows": _log_int(rng, 500, 500_000), "M": rng.choice([64, 128, 256, 512]),
                "spread": rng.random() < 0.5}
    if kind == "sweep":
        precision = rng.choice(["fp64", "fp64", "mixed", "fp32"])
        return {"kind": kind, "n": _log_int(rng, 6, 36), "M": rng.choice([8, 24, 64, 100, 128, 256]),
                "G": rng.choice([1, 1, 2, 3, 4]), "precision": precision,
                "item_geometry": precision != "fp64" and rng.random() < 0.5}
    if kind == "coupled":
        return {"kind": kind, "n": _log_int(rng, 8, 36), "M": rng.choice([64, 128, 256]), "G": rng.choice([1, 2, 4]),
                "form": rng.choice(["plain", "chosen"]), "steps": rng.randint(1, 3)}
    if kind == "compton":
        return {"kind": kind, "cells": _log_int(rng, 1, 290), "M": rng.choice([26, 64, 100, 195, 256])}
    return {"kind": "ray", "n_box": _log_int(rng, 4, 48), "n_sphere": _log_int(rng, 8, 64),
            "mode": rng.choice([rt.SURFACE, rt.INNER, rt.ROCHE]), "frame": rng.randint(0, 59)}


# ------------------------------------------------------------------------------------------------ inputs

@functools.lru_cache(maxsize=2)
def _mesh(problem, nx, ny, nz):
    if problem == "tube":
        return meshes.kuhn_box(nx, ny, nz, hi=(1.0, ny / nx, nz / nx), jitter=0.15, seed=7)
    nozzle = max(0.1, 5.0 / nx)  # coarse meshes widen the nozzle so that it holds some faces
    return meshes.kuhn_box(nx, ny, nz, lo=(-1, -1, -1), hi=(1, 1, 1), jitter=0.15, seed=2024, inflow_radius=nozzle,
                           inflow_code=-3)


def _case_mesh(case):
    if case["kind"] == "hydro":
        return _mesh(case["problem"], case["nx"], case["ny"], case["nz"])
    return _mesh("jet", case["n"], case["n"], case["n"])


def _primitives(m, problem, seed):
    """Initial primitives: the shock tube's two states or the jet's ambient gas, perturbed cell by cell."""
    rng = np.random.default_rng(seed)
    W = np.zeros((m.n_cells, 5))
    if problem == "tube":
        left = m.cell_center[:, 0] < 0.5
        W[:, 0], W[:, 4] = np.where(left, 10.0, 1.0), np.where(left, 13.33, 0.01)
    else:
        W[:, 0], W[:, 4] = 1.0, 1e-3
    W[:, 0] *= 1 + 0.2 * rng.uniform(-1, 1, m.n_cells)
    W[:, 4] *= 1 + 0.2 * rng.uniform(-1, 1, m.n_cells)
    W[:, 1:4] = 0.02 * rng.uniform(-1, 1, (m.n_cells, 3))
    return torch.tensor(W, device=DEV)


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _log_uniform(gen, lo, hi, *shape):
    return 10 ** (lo + (hi - lo) * torch.rand(*shape, generator=gen, device=DEV, dtype=torch.float64))


def _c2p_states(n, seed):
    """Primitives with rho in [1e-4, 1e2], p / rho in [1e-6, 1e2] and Lorentz factors in [1, 50], log-uniform."""
    g = _gen(seed)
    rho = _log_uniform(g, -4, 2, n)
    p = rho * _log_uniform(g, -6, 2, n)
    v = torch.sqrt(1 - _log_uniform(g, 0, math.log10(50.0), n) ** -2)
    u = torch.randn(n, 3, generator=g, device=DEV, dtype=torch.float64)
    u = u / u.norm(dim=1, keepdim=True) * v[:, None]
    return torch.cat([rho[:, None], u, p[:, None]], 1)


def _intensity(case, seed):
    """Lognormal intensities [rows][M]; "spread": 16 groups over 12 decades."""
    rows, M, g = case["rows"], case["M"], _gen(seed)
    spread = case.get("spread", False)
    dt = torch.float32 if case["kind"] == "tc" else torch.float64
    I = torch.randn(rows, M, generator=g, device=DEV, dtype=dt).mul_(1.0 if spread else 0.5).exp_()
    if spread:
        group = torch.arange(rows, device=DEV) % 16
        I *= (10.0 ** (-6.0 + 12.0 * group / 15.0)).to(dt)[:, None]
    return I


def _sweep_inputs(case, m, seed):
    dt = torch.float64 if case["precision"] == "fp64" else torch.float32
    g, G = _gen(seed), case["G"]
    alpha = _log_uniform(g, -1, 1.5, m.n_cells)
    return [t.to(dt).contiguous() for t in (alpha, 0.5 * alpha, _log_uniform(g, -2, 0, m.n_cells, G),
                                            _log_uniform(g, -3, -1, m.n_cells * G, case["M"]))]


def _compton_inputs(case, seed):
    cells, g = case["cells"], _gen(seed)
    shape = torch.exp(-((torch.arange(100, device=DEV, dtype=torch.float64) - 60.0) / 25.0) ** 2) + 0.05
    I = torch.exp(0.5 * torch.randn(cells, case["M"], 100, generator=g, device=DEV, dtype=torch.float64)) * shape
    u = torch.randn(cells, 3, generator=g, device=DEV, dtype=torch.float64)
    speed = torch.tensor(SPEEDS, device=DEV, dtype=torch.float64)[torch.arange(cells, device=DEV) % len(SPEEDS)]
    return I.contiguous(), (u / u.norm(dim=1, keepdim=True) * speed[:, None]).contiguous()


def _surface(n_box, n_sphere, seed):
    """Ids and triangles of the outer box's boundary and a rough sphere around the accretor (1, 0, 0)."""
    rng = np.random.default_rng(seed)
    lo, hi = np.array([0.43, -0.35, -0.25]), np.array([1.33, 0.35, 0.25])
    a, b = (x.ravel() for x in np.meshgrid(np.arange(n_box), np.arange(n_box), indexing="ij"))
    tris = []
    for ax in range(3):
        u, v = [x for x in range(3) if x != ax]
        for side in (lo, hi):
            corner = []
            for da, db in ((0, 0), (1, 0), (1, 1), (0, 1)):
                p = np.empty((n_box * n_box, 3))
                p[:, ax] = side[ax]
                p[:, u] = lo[u] + (hi[u] - lo[u]) * (a + da) / n_box
                p[:, v] = lo[v] + (hi[v] - lo[v]) * (b + db) / n_box
                corner.append(p)
            tris += [np.concatenate(corner[:3], 1), np.concatenate([corner[0], corner[2], corner[3]], 1)]
    th, ph = np.meshgrid(np.linspace(0, np.pi, n_sphere + 1), np.linspace(0, 2 * np.pi, 2 * n_sphere + 1),
                         indexing="ij")
    r = 0.08 * (1 + 0.05 * rng.uniform(-1, 1, th.shape))
    r[0], r[-1], r[:, -1] = 0.08, 0.08, r[:, 0]
    P = np.stack([1 + r * np.sin(th) * np.cos(ph), r * np.sin(th) * np.sin(ph), r * np.cos(th)], -1)
    p00, p10, p11, p01 = (x.reshape(-1, 3) for x in (P[:-1, :-1], P[1:, :-1], P[1:, 1:], P[:-1, 1:]))
    abc = np.concatenate(tris + [np.concatenate([p00, p10, p11], 1), np.concatenate([p00, p11, p01], 1)])
    return rng.permutation(4 * len(abc))[:len(abc)].astype(np.int32), abc


def _p2c(W, gamma):
    rho, v, p = W[:, 0], W[:, 1:4], W[:, 4]
    lor2 = 1 / (1 - (v * v).sum(1))
    w = (rho + gamma / (gamma - 1) * p) * lor2
    return torch.cat([(rho * lor2.sqrt())[:, None], w[:, None] * v, (w - p)[:, None]], 1)


# ------------------------------------------------------------------------------------------------ cases

def _grid(m, gamma, jet):
    grid = rhllc.Grid(m, eos=rhllc.EOS_IDEAL, gamma=gamma)
    if jet:
        grid.set_boundary(-3, rhllc.BC_FIXED, JET_INFLOW)
    return grid


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind in ("hydro", "coupled"):
        m = _case_mesh(case)
        jet = case.get("problem", "jet") == "jet"
        gamma = GAMMA_JET if jet else GAMMA_TUBE
        s["grid"] = _grid(m, gamma, jet)
        s["W"] = _primitives(m, "jet" if jet else "tube", seed)
        s["U"] = _p2c(s["W"], gamma).contiguous()
        s["W_out"], s["U_out"] = torch.empty_like(s["W"]), torch.empty_like(s["U"])
        s["tau"] = CFL * m.h_min
        if kind == "coupled":
            plain = case["form"] == "plain"
            s["dg"] = illum.DirectionGrid(meshes.fibonacci_directions(case["M"]))
            s["guess"] = None
            if not plain:
                n = min(65536, m.n_cells // 128 * 128)
                s["guess"] = LearnedGuess(seed=1)
                s["guess"].train(s["U"][:n].contiguous(), s["W"][:n, 4].contiguous(), epochs=2, batch=min(4096, n))
            sweep = illum.TransportSweep(s["grid"], s["dg"], groups=case["G"], precision="fp64" if plain else "mixed",
                                         dirs_per_batch=128 if plain else 256, item_geometry=not plain)
            s["step"] = rad_rhd.RadRHDStep(sweep, em=rad_rhd.emission(*JET_EMISSION),
                                           scatter="fp64" if plain else "f16x3", guess=s["guess"])
    elif kind == "con2prim":
        s["U"] = _p2c(_c2p_states(case["n"], seed), GAMMA_JET).contiguous()
        s["W"] = torch.empty_like(s["U"])
    elif kind in ("scatter", "tc"):
        s["dg"] = illum.DirectionGrid(meshes.fibonacci_directions(case["M"]))
        s["I"] = _intensity(case, seed)
        s["S"] = torch.empty_like(s["I"])
        if kind == "tc":
            s["tc"] = illum.ScatterTC(s["dg"], case["form"])
    elif kind == "sweep":
        m = _case_mesh(case)
        s["grid"] = _grid(m, GAMMA_JET, True)
        s["dg"] = illum.DirectionGrid(meshes.fibonacci_directions(case["M"]))
        s["sweep"] = illum.TransportSweep(s["grid"], s["dg"], groups=case["G"], precision=case["precision"],
                                          item_geometry=case["item_geometry"])
        s["inputs"] = _sweep_inputs(case, m, seed)
        s["I"] = torch.empty_like(s["inputs"][3])
    elif kind == "compton":
        s["dg"] = illum.DirectionGrid(meshes.fibonacci_directions(case["M"]))
        s["I"], s["vel"] = _compton_inputs(case, seed)
        s["S"] = torch.empty_like(s["I"])
    else:
        ids, abc = _surface(case["n_box"], case["n_sphere"], seed)
        s["tracer"] = rt.RayTracer(rt.face_cells(ids, abc))
        s["rays"] = torch.tensor(rt.MakeRays(case["frame"]), device=DEV)
        s["codes"] = torch.empty(len(s["rays"]), dtype=torch.int32, device=DEV)
        s["values"] = torch.rand(len(abc), generator=_gen(seed), device=DEV, dtype=torch.float64)
    return s


def run(s):
    kind = s["kind"]
    if kind in ("hydro", "coupled"):
        grid = s["grid"]
        grid.set_state(s["W"], s["U"])
        for _ in range(s["case"]["steps"]):
            if kind == "hydro":
                rhllc.Hllc3dStab(s["tau"], grid)
            else:
                s["step"](s["tau"])
        L.check(L.lib.rrhd_get_state(grid.handle, L.ptr(s["W_out"]), L.ptr(s["U_out"]), 5, L.RRHD_DEVICE))
        return {"W": s["W_out"], "U": s["U_out"]}
    if kind == "con2prim":
        rhllc.GetPhysValueStab(s["U"], s["W"], gamma=GAMMA_JET, fallback=True,
                               stream=torch.cuda.current_stream().cuda_stream)
        return {"W": s["W"]}
    if kind == "scatter":
        S = illum.CalculateIntScattering(s["dg"], s["I"], s["S"])
        E, F, T = illum.CalculateAllParam(s["dg"], s["I"])
        return {"S": S, "E": E, "F": F, "T": T}
    if kind == "tc":
        S, moments = s["tc"](s["I"], s["S"])
        return {"S": S, "moments": moments}
    if kind == "sweep":
        return {"I": illum.CalculateIllum(s["sweep"], *s["inputs"], s["I"])}
    if kind == "compton":
        return {"S": illum.FullSpectrumScattering(s["dg"], s["I"], s["vel"], s["S"])}
    codes = s["tracer"].trace(s["rays"], s["case"]["mode"], s["codes"])
    image, curve = s["tracer"].image(codes, s["values"])
    return {"codes": codes, "image": image, "curve": curve}


def _cells_faces(case):
    if "nx" in case:
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
    else:
        nx = ny = nz = case["n"]
    return 6 * nx * ny * nz, 12 * nx * ny * nz + 2 * (nx * ny + ny * nz + nx * nz)


def work(case):
    """Bytes: each input read once and each output written once.  Operations: the multiply-adds of the contraction,
    or an estimate of the path's arithmetic per cell, face, term or ray (stated beside it)."""
    kind = case["kind"]
    if kind in ("hydro", "coupled"):
        N, F = _cells_faces(case)
        # a step: state read and written (160 B), cell records (25 B) and face records (40 B); per cell two face
        # fluxes and a primitive recovery, about 1200 operations
        step_bytes, step_flops = 185.0 * N + 40.0 * F, 1200.0 * N
        if kind == "coupled":
            M, G = case["M"], case["G"]
            b = 8 if case["form"] == "plain" else 4
            # the sweep reads S and writes I, the scattering reads I and writes S
            step_bytes += 4.0 * b * N * M * G
            # sweep: about 60 operations per (cell, direction) and 60 per group; contraction: 2 M per element
            step_flops += N * M * (60.0 + 60.0 * G) + 2.0 * N * G * M * (M + 10)
        return {"bytes": case["steps"] * step_bytes, "flops": case["steps"] * step_flops}
    if kind == "con2prim":  # about 40 operations a Newton iteration, three iterations, 30 outside the loop
        return {"bytes": 80.0 * case["n"], "flops": 150.0 * case["n"]}
    if kind in ("scatter", "tc"):
        n = float(case["rows"]) * case["M"]
        return {"bytes": n * (16 if kind == "scatter" else 8) + case["rows"] * (104 if kind == "scatter" else 64),
                "flops": 2.0 * n * (case["M"] + 10)}
    if kind == "sweep":
        N, F = _cells_faces(case)
        b = 8 if case["precision"] == "fp64" else 4
        M, G = case["M"], case["G"]
        return {"bytes": 2.0 * b * N * M * G + N * (20 * b + 16) + b * N * (2 + G), "flops": N * M * (60.0 + 60.0 * G)}
    if kind == "compton":  # 32 operations per (cell, output direction, bin, input direction)
        n = float(case["cells"]) * case["M"] * 100
        return {"bytes": 16.0 * n, "flops": 32.0 * n * case["M"]}
    triangles = 12 * case["n_box"] ** 2 + 4 * case["n_sphere"] ** 2
    rays = rt.PIXELS[0] * rt.PIXELS[1]
    # each ray against the two triangles it meets: 50 operations a test
    return {"bytes": rays * (48.0 + 4 + 4 + 8) + triangles * (80.0 + 8), "flops": rays * 100.0}


# ------------------------------------------------------------------------------------------------ 64-bit values

def exact(case, seed):
    kind = case["kind"]
    if kind == "hydro":
        return _exact_hydro(case, seed)
    if kind == "con2prim":
        U = _p2c(_c2p_states(case["n"], seed), GAMMA_JET)
        return {"W": _c2p(U, GAMMA_JET)}
    if kind in ("scatter", "tc"):
        return _exact_scatter(case, seed)
    if kind == "sweep":
        return _exact_sweep(case, seed)
    if kind == "compton":
        return _exact_compton(case, seed)
    # coupled: the state of a whole trajectory (its intensity carries over from pass to pass);
    # ray: whole numbers, and an image looked up by them
    return None


def _c2p(U, gamma):
    """Newton iteration for the pressure, forty steps or until it stands."""
    D, E = U[:, 0], U[:, 4]
    m2 = (U[:, 1:4] ** 2).sum(1)
    gg = gamma / (gamma - 1)
    floor = torch.sqrt(m2 / (1 - 1e-12)) - E
    p = torch.maximum(torch.clamp(torch.sqrt(m2) - E, min=0.0), floor)
    for _ in range(40):
        a = E + p
        lor2 = 1 / (1 - m2 / (a * a))
        lor = lor2.sqrt()
        h = 1 + gg * p * lor / D
        y = D * h * lor - a
        dy = gg * lor2 - m2 * lor2 * lor / a ** 3 * (gg * p * lor + D * h) - 1
        new = torch.maximum(p - y / dy, floor)
        still = bool(((new - p).abs() <= 1e-15 * E).all())
        p = new
        if still:
            break
    a = E + p
    lor = torch.sqrt(a * a / (a * a - m2))
    return torch.cat([(D / lor)[:, None], U[:, 1:4] / a[:, None], p[:, None]], 1)


def _exact_hydro(case, seed):
    m = _case_mesh(case)
    jet = case["problem"] == "jet"
    gamma = GAMMA_JET if jet else GAMMA_TUBE
    gg = gamma / (gamma - 1)
    cu = lambda a: torch.tensor(a, device=DEV)  # noqa: E731
    n, area = cu(m.face_n), cu(m.face_area)
    left, right = cu(m.face_id_l).long(), cu(m.face_id_r).long()
    edge, inflow = right < 0, right == -3
    right = torch.where(edge, left, right)
    faces = cu(m.cell_faces).long()
    sign = torch.stack([(cu(m.cell_sign.astype(np.int64)) >> j & 1) * 2 - 1 for j in range(4)], 1).double()
    rate = CFL * m.h_min / cu(m.cell_volume)
    Win = torch.tensor([JET_INFLOW], device=DEV, dtype=torch.float64)
    Uin = _p2c(Win, gamma)

    def side(W, U):
        vn, vv = (W[:, 1:4] * n).sum(1), (W[:, 1:4] ** 2).sum(1)
        cs2 = gamma * W[:, 4] / (W[:, 0] + gg * W[:, 4])
        root = torch.sqrt(cs2 * (1 - vn * vn - (vv - vn * vn) * cs2) * (1 - vv))
        den = 1 - vv * cs2
        return vn, (U[:, 1:4] * n).sum(1), (vn * (1 - cs2) - root) / den, (vn * (1 - cs2) + root) / den

    W = _primitives(m, case["problem"], seed)
    U = _p2c(W, gamma)
    for _ in range(case["steps"]):
        Wl, Ul, Wr, Ur = W[left], U[left], W[right], U[right]
        if jet:
            Wr, Ur = torch.where(inflow[:, None], Win, Wr), torch.where(inflow[:, None], Uin, Ur)
        vl, ml, cl0, cl1 = side(Wl, Ul)
        vr, mr, cr0, cr1 = side(Wr, Ur)
        lo, hi = torch.minimum(cl0, cr0), torch.maximum(cl1, cr1)
        AL, AR = lo * Ul[:, 4] - ml, hi * Ur[:, 4] - mr
        BL, BR = lo * ml - ml * vl - Wl[:, 4], hi * mr - mr * vr - Wr[:, 4]
        a, b, c = AR * lo - AL * hi, AL + BL * hi - AR - BR * lo, BR - BL
        us = c / (-0.5 * (b + torch.where(b < 0, -1.0, 1.0) * torch.sqrt(b * b - 4 * a * c)))
        ps = (AL * us - BL) / (1 - us * lo)
        star = (lo < 0) & (hi > 0)
        use_r = torch.where(star, ~(us >= 0), lo < 0)
        pick = lambda x, y: torch.where(use_r if x.dim() == 1 else use_r[:, None], y, x)  # noqa: E731
        Us, vn, mn, p, lam = pick(Ul, Ur), pick(vl, vr), pick(ml, mr), pick(Wl[:, 4], Wr[:, 4]), pick(lo, hi)
        D, E = Us[:, 0], Us[:, 4]
        St = Us[:, 1:4] - mn[:, None] * n
        k = (lam - vn) / (lam - us) - 1
        sn = (lam * (E + ps) - mn) * us / (lam - us)
        zero = torch.zeros_like(D)
        fD = D * vn + torch.where(star, lam * D * k, zero)
        fn = mn * vn + p + torch.where(star, lam * (sn - mn), zero)
        fE = mn + torch.where(star, sn - mn, zero)
        ft = St * (vn + torch.where(star, lam * k, zero))[:, None]
        flux = torch.cat([fD[:, None], ft + fn[:, None] * n, fE[:, None]], 1) * area[:, None]
        U = U - rate[:, None] * (flux[faces] * sign[:, :, None]).sum(1)
        W = _c2p(U, gamma)
    return {"W": W, "U": U}


def _exact_scatter(case, seed):
    d = meshes.fibonacci_directions(case["M"])
    w, a = torch.tensor(d.dirs, device=DEV), torch.tensor(d.areas, device=DEV) / d.full_area
    I = _intensity(case, seed)
    K = a[:, None] * 0.75 * (1 + (w @ w.T) ** 2)
    outer = (w[:, :, None] * w[:, None, :]).reshape(-1, 9)
    basis = a[:, None] * torch.cat([torch.ones_like(w[:, :1]), w, outer], 1)
    S = torch.empty(I.shape, dtype=torch.float64, device=DEV)
    mom = torch.empty(len(I), 13, dtype=torch.float64, device=DEV)
    for r in range(0, len(I), 65536):
        block = I[r:r + 65536].double()
        S[r:r + 65536] = block @ K
        mom[r:r + 65536] = block @ basis
    if case["kind"] == "scatter":
        return {"S": S, "E": mom[:, 0].clone(), "F": mom[:, 1:4].clone(), "T": mom[:, 4:].reshape(-1, 3, 3).clone()}
    six = torch.zeros(len(I), 16, dtype=torch.float64, device=DEV)
    six[:, :4] = mom[:, :4]
    six[:, 4:10] = mom[:, [4, 5, 6, 8, 9, 12]]
    return {"S": S, "moments": six}


def _exact_sweep(case, seed):
    """Cells in upwind order, all directions at once: each front's pairs (cell, direction) in one set of tensors."""
    m, M, G = _case_mesh(case), case["M"], case["G"]
    N, F = m.n_cells, m.n_faces
    cu = lambda a: torch.tensor(a, device=DEV)  # noqa: E731
    w = cu(meshes.fibonacci_directions(M).dirs)
    alpha, betta, Q, S = (t.double() for t in _sweep_inputs(case, m, seed))
    S = S.reshape(N, G, M)
    k = alpha + betta
    faces = cu(m.cell_faces).long()
    sign = torch.stack([(cu(m.cell_sign.astype(np.int64)) >> j & 1) * 2 - 1 for j in range(4)], 1).double()
    normal = cu(m.face_n)[faces] * sign[:, :, None]
    area = cu(m.face_area)[faces]
    height = 3 * cu(m.cell_volume)[:, None] / area
    own = torch.arange(N, device=DEV)[:, None]
    nbr = cu(m.face_id_l).long()[faces]
    nbr = torch.where(nbr == own, cu(m.face_id_r).long()[faces], nbr)
    out = torch.empty(N, G, M, dtype=torch.float64, device=DEV)
    indeg = torch.zeros(N * M, dtype=torch.int32, device=DEV)
    for j in range(4):
        indeg += (((normal[:, j] @ w.T) < 0) & (nbr[:, j:j + 1] >= 0)).reshape(-1).int()
    fv = torch.zeros(F * M, G, dtype=torch.float64, device=DEV)
    front = torch.nonzero(indeg == 0).reshape(-1)
    vertex = torch.arange(4, device=DEV)
    lam = torch.full((4, 4), 1.0 / 6.0, device=DEV, dtype=torch.float64)  # node's weight of vertex f, node of vertex v
    lam[vertex, vertex] = 2.0 / 3.0
    while len(front):
        c, d = front // M, front % M
        cos = (normal[c] * w[d][:, None, :]).sum(2)
        inward, outward = cos < 0, cos > 0
        reach = torch.where(inward, height[c] / -cos, math.inf)
        t, h = (reach[:, None, :] * lam).min(2)  # per node of vertex v: distance back and in-face
        slot = faces[c] * M + d[:, None]
        value = torch.where((inward & (nbr[c] >= 0))[:, :, None], fv[slot], 0.0)  # boundaries let nothing in
        rhs = (alpha[c, None] * Q[c] + betta[c, None] * S[c, :, d]) / k[c, None]
        start = torch.gather(value, 1, h[:, :, None].expand(-1, -1, G))
        traced = torch.isfinite(t)[:, :, None]
        node = torch.exp(-k[c, None] * torch.where(torch.isfinite(t), t, 0.0))[:, :, None] * (
            torch.where(traced, start, 0.0) - rhs[:, None, :]) + rhs[:, None, :]
        leaving = (node.sum(1, keepdim=True) - node) / 3
        value = torch.where(outward[:, :, None], leaving, value)
        fv[slot[outward]] = leaving[outward]
        weight = area[c]
        mean = (value * weight[:, :, None]).sum(1) / weight.sum(1, keepdim=True)
        out[c, :, d] = torch.where((c == N - 1)[:, None], value.mean(1), mean)
        down = (nbr[c] * M + d[:, None])[outward & (nbr[c] >= 0)]
        indeg.index_add_(0, down, torch.full_like(down, -1, dtype=torch.int32))
        front = torch.unique(down[indeg[down] == 0])
    return {"I": out.reshape(N * G, M)}


def _exact_compton(case, seed):
    """The frequency-coupled Compton sum term by term, CGS constants as the reference code writes them."""
    I, vel = _compton_inputs(case, seed)
    ds = meshes.fibonacci_directions(case["M"])
    w, a = torch.tensor(ds.dirs, device=DEV), torch.tensor(ds.areas, device=DEV)
    light = 3 * 1e10
    eps_of = (6.62 * 1e-27) / (((9.109383701528 * 1e-28) * light) * light)
    coef = ((2 * math.pi) * (2.8179403 * 1e-13)) * (2.8179403 * 1e-13)
    idx = torch.arange(101, device=DEV, dtype=torch.float64)
    edge = 1e24 * torch.exp(-((100 - idx) * (100 - idx)) / 350.0)
    edge[0] = 0.0
    frq = (0.5 * (edge[1:] + edge[:-1]))[None, :, None]  # [1][bin][1]
    low, high = 0.5 * (edge[1] + edge[0]), edge[99]
    mu = (w[:, None, 0] * w[None, :, 0] + w[:, None, 1] * w[None, :, 1]) + w[:, None, 2] * w[None, :, 2]
    S = torch.empty_like(I)
    every = torch.arange(case["M"], device=DEV)
    for i in range(len(I)):
        v3 = vel[i]
        v2 = (v3[0] * v3[0] + v3[1] * v3[1]) + v3[2] * v3[2]
        moving = float(v2) > 1 / light
        v = torch.sqrt(v2) if moving else torch.zeros_like(v2)
        if float(v) > 1 / light:
            lor = 1 / torch.sqrt(1 - v2)
            cf = ((v3[0] * w[:, 0] + v3[1] * w[:, 1]) + v3[2] * w[:, 2]) / v
        for k0 in range(0, case["M"], 64):  # output directions in blocks
            cos = mu[k0:k0 + 64, None, :]
            if float(v) > 1 / light:
                f1 = frq * (1 - v * cf[k0:k0 + 64, None, None]) / (
                    1 + eps_of * frq / lor * (1 - cos) - v * cf[None, None, :])
                forward = None
            else:
                f1 = frq / (1 + eps_of * frq * (1 - cos))
                forward = (cos > 0.99999999).expand_as(f1)
                f1 = torch.where(forward, frq.expand_as(f1), f1)
            ratio = f1 / frq
            G = coef * ratio * ratio * (ratio + 1 / ratio + cos * cos - 1) / ratio
            if forward is not None:
                G = torch.where(forward, 2.0 * coef, G)
            keep = ~(f1 < low) & ~(f1 > high)
            bin_ = 100 - torch.floor(torch.sqrt(torch.clamp(-350.0 * torch.log(f1 / 1e24), min=0.0)) + 1).clamp(0, 100)
            Iv = I[i][every[None, None, :], bin_.long().clamp(0, 99)]
            S[i, k0:k0 + 64] = (G * torch.where(keep, Iv, 0.0) * a).sum(2) / ds.full_area
    return {"S": S}
