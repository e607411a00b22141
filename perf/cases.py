"""Performance cases: the work a user of this package has it do, through its public entry points.

``listed()`` names the fixed cases and ``draw(rng)`` gives further ones of the
same ranges.  ``prepare`` makes, from a seed, what a program holds before the
call (meshes, sheets, stencils, schedules, the rotation index), ``run`` is one
call and ``work`` the bytes and operations it cannot do without.  ``exact``
gives the 64-bit result where plain torch can form it in seconds.

Meshes are convex hulls of jittered Fibonacci points, folded radially by
smooth waves (``synthetic.folded_hull`` with a cheaper fold); sheets are
``synthetic.smooth_sheet``.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from cat_surface_gpu_b200 import synthetic
from cat_surface_gpu_b200.dartel_adjoint import dartel_data_term
from cat_surface_gpu_b200.dartel_grid import dartel_step
from cat_surface_gpu_b200.gifti import GiftiMesh
from cat_surface_gpu_b200.gpu_pipeline import register_meshes
from cat_surface_gpu_b200.rotation_feature import compute_rotation_features
from cat_surface_gpu_b200.surf2sphere import (Surf2SphereTopology, run_areal_smoothing_cuda,
                                              run_surf2sphere_preprocess_cuda, surface_area)
from cat_surface_gpu_b200.surface_rotation import (RotationGridIndexDevice, batched_costs, quaternion_matrices,
                                                   uniform_quaternions)
from cat_surface_gpu_b200.surface_stencil import build_surface_stencil, resampling_sphere
from cat_surface_gpu_b200.surface_warp import solve_dartel_maps, solve_dartel_registrations

DEVICE = "cuda"
DTYPES = {"float32": torch.float32, "float64": torch.float64}
MAX_MESH = 61442  # vertices of a hemisphere mesh (122,880 triangles)


def listed():
    return [
        # one Gauss-Newton step on a small sheet: what an interactive caller of the DARTEL operators does;
        # a few dozen launches of a few microseconds each
        {"name": "dartel-step-64x32-f32", "kind": "step", "nx": 64, "ny": 32, "k": 3, "code": 1, "dtype": "float32"},
        # the DARTEL solve of one SurfWarp run at the 256 x 128 sheet (two step maps, float64, replayed graph)
        {"name": "dartel-solve-256x128-f64", "kind": "solve", "nx": 256, "ny": 128, "steps": 2, "dtype": "float64",
         "graph": True},
        # the same at the pipeline's default 512 x 256 sheet; a single run without -avg does not capture a graph
        {"name": "dartel-solve-512x256-f64", "kind": "solve", "nx": 512, "ny": 256, "steps": 2, "dtype": "float64",
         "graph": False},
        # 16 subjects registered to one template in one batched float32 solve
        {"name": "dartel-batch-16x2-f32", "kind": "many", "nx": 256, "ny": 128, "regs": 16, "steps": 2,
         "dtype": "float32", "graph": True},
        # forward and backward of the data term for 16 registrations x 2 maps
        {"name": "data-term-grad-32-f64", "kind": "adjoint", "nx": 256, "ny": 128, "batch": 32, "k": 7,
         "dtype": "float64"},
        # the initial rotation of a registration: 46 seeds, then host-driven Nelder-Mead
        {"name": "rotation-search", "kind": "search", "subdivisions": 6, "refine": True},
        # candidate rotations of two surfaces scored in one launch, two features each
        {"name": "rotation-batch", "kind": "rotations", "points": 61442, "more_points": 102400, "candidates": 512, "features": 2},
        # the default rotation feature (depth potential, 1,000 coloured SOR sweeps) of both sides
        {"name": "depth-feature", "kind": "depth", "vertices": MAX_MESH, "subdivisions": 6, "sides": 2,
         "solver": "colored-sor"},
        # the curvature sheets of one surface that feed a DARTEL run
        {"name": "curvature-sheets", "kind": "sheets", "vertices": MAX_MESH, "subdivisions": 6, "nx": 256, "ny": 128,
         "fwhm": 5.0 / 9.0, "steps": 2},
        # the 4,999 ordered area-smoothing sweeps of a hemisphere
        {"name": "sweeps-hemisphere", "kind": "sweeps", "vertices": MAX_MESH, "stop_at": 10, "arithmetic": "cat",
         "dtype": "float32"},
        # stages 1-5 of a hemisphere (smoothing, inflation, finger smoothing, ellipsoid)
        {"name": "stages-hemisphere", "kind": "stages", "vertices": MAX_MESH, "stop_at": 5},
        # a whole registration: stencils, features, rotation, two runs, -avg, warp
        {"name": "register-hemisphere", "kind": "register", "vertices": MAX_MESH, "target_vertices": MAX_MESH, "nx": 256, "ny": 128,
         "steps": 2, "runs": 2, "avg": True},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["step", "solve", "many", "adjoint", "search", "rotations", "depth", "sheets", "sweeps", "stages",
                       "register"])
    dtype = rng.choice(["float32", "float64"])
    if kind == "step":
        nx = rng.choice([32, 64, 128, 256])
        return {"kind": kind, "nx": nx, "ny": _log_int(rng, nx // 4, nx), "k": rng.randint(0, 5),
                "code": rng.randint(0, 1), "dtype": dtype}
    if kind == "solve":
        nx = rng.choice([64, 128, 256, 512])
        return {"kind": kind, "nx": nx, "ny": rng.randint(nx // 2 - nx // 16, nx // 2), "steps": rng.randint(1, 3),
                "dtype": dtype, "graph": rng.random() < 0.5}
    if kind == "many":
        nx = rng.choice([64, 128, 256])
        return {"kind": kind, "nx": nx, "ny": rng.randint(nx // 2 - nx // 16, nx // 2), "regs": _log_int(rng, 2, 16),
                "steps": rng.randint(1, 2), "dtype": dtype, "graph": rng.random() < 0.5}
    if kind == "adjoint":
        nx = _log_int(rng, 32, 256)
        return {"kind": kind, "nx": nx, "ny": rng.randint(nx // 2, nx // 2 + 9), "batch": _log_int(rng, 1, 32),
                "k": rng.randint(0, 8), "dtype": dtype}
    if kind == "search":
        return {"kind": kind, "subdivisions": rng.choice([5, 6]), "refine": rng.random() < 0.75}
    if kind == "rotations":
        points = _log_int(rng, 2562, 102400)
        more = _log_int(rng, 2562, 102400) if rng.random() < 0.5 else 0
        most = (61442 + 102400) * 512 // (points + more)
        return {"kind": kind, "points": points, "more_points": more, "candidates": _log_int(rng, 1, min(2048, most)),
                "features": rng.randint(1, 2)}
    if kind == "depth":
        return {"kind": kind, "vertices": _log_int(rng, 2562, MAX_MESH), "subdivisions": rng.choice([4, 5, 6]),
                "sides": rng.randint(1, 2), "solver": rng.choice(["colored-sor", "colored-sor", "pcg"])}
    if kind == "sheets":
        nx = rng.choice([128, 256, 512])
        return {"kind": kind, "vertices": _log_int(rng, 2562, MAX_MESH), "subdivisions": rng.choice([5, 6]), "nx": nx,
                "ny": nx // 2, "fwhm": rng.choice([5.0 / 3.0, 5.0 / 9.0, 5.0 / 27.0]), "steps": rng.randint(2, 3)}
    if kind == "sweeps":
        mode = rng.choice(["cat", "cat", "cat", "fp32", "fp64"])
        return {"kind": kind, "vertices": _log_int(rng, 2562, MAX_MESH), "stop_at": rng.randint(6, 10),
                "arithmetic": "fp32" if mode == "fp32" else "cat", "dtype": "float64" if mode == "fp64" else "float32"}
    if kind == "stages":
        return {"kind": kind, "vertices": _log_int(rng, 2562, MAX_MESH), "stop_at": rng.randint(1, 5)}
    nx = rng.choice([64, 128, 256])
    return {"kind": kind, "vertices": _log_int(rng, 2562, 40962), "target_vertices": _log_int(rng, 2562, 40962),
            "nx": nx, "ny": nx // 2, "steps": rng.randint(1, 2), "runs": rng.randint(1, 2), "avg": rng.random() < 0.5}


# ------------------------------------------------------------------ inputs


def _waves(points, rng, low, high, std, count=32):
    """A smooth random function of unit points: plane waves of wave number low..high, standard deviation ~ std."""

    direction = rng.normal(size=(count, 3))
    direction /= np.linalg.norm(direction, axis=1, keepdims=True)
    phase = (points @ (direction * rng.uniform(low, high, (count, 1))).T) + rng.uniform(0, 2 * np.pi, count)
    return np.cos(phase).sum(axis=1) * (std * math.sqrt(2.0 / count))


def _mesh(n, rng):
    """A folded hull and its sphere: (surface float32 [n, 3] mm, faces int32, sphere float32 [n, 3])."""

    points = synthetic.fibonacci_points(n, rng)
    faces = synthetic.hull_faces(points)
    r = 70.0 * np.exp(_waves(points, rng, 8.0, 40.0, 0.3))
    return (points * r[:, None]).astype(np.float32), faces, (100.0 * points).astype(np.float32)


def _sheets(count, ny, nx, seed):
    return np.stack([synthetic.smooth_sheet(ny, nx, seed + i) for i in range(count)])


def _unit_features(points, rng, count):
    values = np.stack([_waves(points, rng, 3.0, 12.0, 1.0) for _ in range(count)])
    return (values - values.mean(axis=1, keepdims=True)) / values.std(axis=1, keepdims=True)


def _cuda(array, dtype=None):
    return torch.as_tensor(np.ascontiguousarray(array), dtype=dtype, device=DEVICE)


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    base = int(rng.integers(1 << 30))
    state = {"case": case}
    if kind == "step":
        nx, ny, dtype = case["nx"], case["ny"], DTYPES[case["dtype"]]
        maps = _sheets(4, ny, nx, base)
        state.update(source=_cuda(maps[0], dtype), target=_cuda(maps[1], dtype),
                     velocity=_cuda(maps[2:] - 0.5, dtype), dtype=dtype)
    elif kind in ("solve", "many"):
        nx, ny, dtype = case["nx"], case["ny"], DTYPES[case["dtype"]]
        steps, regs = case["steps"], case.get("regs", 1)
        source = _sheets(regs * steps, ny, nx, base).reshape(regs, steps, ny, nx)
        target = np.broadcast_to(_sheets(steps, ny, nx, base + 7919), source.shape)  # one template
        if kind == "solve":
            source, target = source[0], target[0]
        state.update(source=_cuda(source, dtype), target=_cuda(target, dtype), dtype=dtype)
    elif kind == "adjoint":
        nx, ny, dtype, batch = case["nx"], case["ny"], DTYPES[case["dtype"]], case["batch"]
        velocity = _sheets(2 * batch, ny, nx, base).reshape(batch, 2, ny, nx) * 8.0 - 4.0
        state.update(source=_cuda(_sheets(batch, ny, nx, base + 3001), dtype),
                     target=_cuda(_sheets(batch, ny, nx, base + 6007), dtype), velocity=_cuda(velocity, dtype))
    elif kind == "search":
        points, faces = resampling_sphere(case["subdivisions"])
        angles = rng.uniform(-0.4, 0.4, 3)
        source = points @ _euler(angles).T
        wave_seed = int(rng.integers(1 << 30))
        target_values = _waves(points, np.random.default_rng(wave_seed), 3.0, 12.0, 1.0)
        source_values = _waves(source, np.random.default_rng(wave_seed), 3.0, 12.0, 1.0)
        source_values = source_values + _waves(points, rng, 10.0, 20.0, 0.1)
        index = RotationGridIndexDevice.build(points, faces, device=DEVICE)
        state.update(index=index, inputs=index.prepare_cost_inputs(
            points.astype(np.float32), _minmax_np(source_values), _minmax_np(target_values)))
    elif kind == "rotations":
        points, faces = resampling_sphere(6)
        index = RotationGridIndexDevice.build(points, faces, device=DEVICE)
        target_values = _unit_features(points, rng, case["features"])
        inputs, matrices = [], []
        for i, n in enumerate(_point_counts(case)):
            source = synthetic.fibonacci_points(n, rng)
            inputs.append(index.prepare_cost_inputs(source.astype(np.float32),
                                                    _unit_features(source, rng, case["features"]), target_values))
            matrices.append(quaternion_matrices(uniform_quaternions(case["candidates"], base + i)))
        state.update(indices=[index] * len(inputs), inputs=inputs, matrices=matrices)
    elif kind in ("depth", "sheets"):
        stencils, surfaces = [], []
        for _ in range(case.get("sides", 1)):
            surface, faces, sphere = _mesh(case["vertices"], rng)
            stencil = build_surface_stencil(sphere, faces, nx=case.get("nx", 64), ny=case.get("ny", 32),
                                            subdivisions=case["subdivisions"], device=DEVICE)
            stencils.append(stencil.to(DEVICE, geometry_dtype=torch.float32))
            surfaces.append(_cuda(surface))
        state.update(stencils=stencils, surfaces=surfaces)
    elif kind in ("sweeps", "stages"):
        surface, faces, sphere = _mesh(case["vertices"], rng)
        if kind == "sweeps":
            # an uneven sphere, as stages 1-5 leave it
            points = sphere.astype(np.float64) / 100.0
            points = points + np.stack([_waves(points, rng, 2.0, 8.0, 0.02) for _ in range(3)], axis=1)
            points /= np.linalg.norm(points, axis=1, keepdims=True)
            surface = (points * 80.0).astype(np.float32)
        mesh = GiftiMesh(surface, faces)
        state.update(vertices=surface, faces=faces, topology=Surf2SphereTopology.plan_only(mesh),
                     area=surface_area(mesh),
                     radius=float(np.sqrt(np.max(np.sum(surface.astype(np.float64) ** 2, axis=1)))))
    else:
        meshes = []
        for n in (case["vertices"], case["target_vertices"]):
            surface, faces, sphere = _mesh(n, rng)
            meshes += [GiftiMesh(surface, faces), GiftiMesh(sphere, faces)]
        state.update(meshes=meshes)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        velocity, metrics = dartel_step(state["source"], state["target"], state["velocity"], k=case["k"],
                                        code=case["code"], device=DEVICE, dtype=state["dtype"])
        return {"velocity": velocity, "metrics": metrics}
    if kind == "solve":
        result = solve_dartel_maps(state["source"], state["target"], device=DEVICE, dtype=state["dtype"],
                                   cuda_graph=case["graph"])
        return {"flow": result.flow, "metrics": result.metrics}
    if kind == "many":
        flows, metrics = solve_dartel_registrations(state["source"], state["target"], device=DEVICE,
                                                    dtype=state["dtype"], cuda_graph=case["graph"])
        return {"flows": flows, "metrics": metrics}
    if kind == "adjoint":
        velocity = state["velocity"].detach().requires_grad_(True)
        energy = dartel_data_term(velocity, state["source"], state["target"], case["k"])
        (grad,) = torch.autograd.grad(energy.sum(), velocity)
        return {"energy": energy.detach(), "grad": grad}
    if kind == "search":
        result = state["index"].search_rotation_prepared(state["inputs"], refine=case["refine"])
        return {"angle": result.angle, "cost": result.cost, "seed_costs": result.seed_costs}
    if kind == "rotations":
        return batched_costs(state["indices"], state["inputs"], matrix_sets=state["matrices"])
    if kind == "depth":
        results = compute_rotation_features(state["stencils"], state["surfaces"],
                                            heat_fwhms=(15.0, 10.0)[:len(state["surfaces"])], solver=case["solver"])
        return [r.values for r in results]
    if kind == "sheets":
        stencil = state["stencils"][0]
        mapped = stencil.resample_vertices(state["surfaces"][0])
        return list(stencil.curvature_type5_to_sheet_many(mapped, _fwhms(case)))
    if kind == "sweeps":
        return run_areal_smoothing_cuda(state["vertices"], state["faces"], state["topology"],
                                        iterations=1000 * (case["stop_at"] - 5), project_every=1000,
                                        radius=state["radius"], device=DEVICE, dtype=DTYPES[case["dtype"]],
                                        arithmetic=case["arithmetic"])[0]
    if kind == "stages":
        return run_surf2sphere_preprocess_cuda(state["vertices"], state["faces"], state["topology"],
                                               stop_at=case["stop_at"], desired_surface_area=state["area"],
                                               device=DEVICE)[0]
    vertices, angle, cost, _ = register_meshes(*state["meshes"], device=DEVICE, steps=case["steps"], runs=case["runs"],
                                               avg=case["avg"], sheet_size=(case["nx"], case["ny"]))
    return {"vertices": vertices, "angle": angle, "cost": cost}


def _point_counts(case):
    return [n for n in (case["points"], case["more_points"]) if n]


def _fwhms(case):
    return tuple(case["fwhm"] / 3.0 ** i for i in range(case["steps"]))


# ------------------------------------------------------------------ work


def _step_flops(points, k, code, cycles=3, nit=3):
    """Operations of one dartel_step: the maps, both squaring chains and the V-cycles' half-sweeps."""

    chain = k * 60 + 60 + (1 + code) * (k * 110 + 40)
    cycle = 2 * nit * 2 * 0.5 * 2 * 30 + 40 + 2 * 30  # relaxation down and up, residual, both transfers
    return points * (chain + cycles * cycle * 4.0 / 3.0)


def work(case):
    kind = case["kind"]
    if kind in ("step", "solve", "many"):
        size = 8 if case["dtype"] == "float64" else 4
        points = case["nx"] * case["ny"]
        if kind == "step":
            return {"bytes": (4 + 2) * points * size, "flops": _step_flops(points, case["k"], case["code"])}
        maps = case["steps"] * case.get("regs", 1)
        flops = sum(3 * _step_flops(points, k, 1) for k in range(6)) * maps
        return {"bytes": (2 * maps + 2 * case.get("regs", 1)) * points * size, "flops": flops}
    if kind == "adjoint":
        points = case["nx"] * case["ny"] * case["batch"]
        size = 8 if case["dtype"] == "float64" else 4
        return {"bytes": (2 + 2 + 2) * points * size, "flops": points * (60 * 2 * case["k"] + 50 + 90 * case["k"])}
    if kind == "search":
        n = 10 * 4 ** case["subdivisions"] + 2
        evaluations = n * (46 + (250 if case["refine"] else 0))
        return {"bytes": n * (12 + 8 + 12 + 8 + 24), "flops": evaluations * 200}
    if kind == "rotations":
        n, targets = sum(_point_counts(case)), 40962
        return {"bytes": n * (12 + 8 * case["features"]) + targets * (12 + 24 + 8 * case["features"]),
                "flops": n * case["candidates"] * 200.0}
    if kind in ("depth", "sheets"):
        n = 10 * 4 ** case["subdivisions"] + 2
        if kind == "depth":
            # 1,000 sweeps over 7-entry rows, and the two heat smoothings
            return {"bytes": case["sides"] * (12 * case["vertices"] + n * (36 + 24 + 8 + 7 * 12)),
                    "flops": case["sides"] * n * 7.0 * 2 * 1100}
        cells = case["nx"] * case["ny"]
        return {"bytes": 12 * case["vertices"] + n * (36 + 12 + 24 + 28) + cells * 36 + 8 * cells * case["steps"],
                "flops": n * 7.0 * 6 * 300}
    if kind in ("sweeps", "stages"):
        n = case["vertices"]
        faces = 2 * n - 4
        sweeps = 1000 * (case["stop_at"] - 5) - 1 if kind == "sweeps" else 60 * case["stop_at"]
        return {"bytes": 24 * n + 12 * faces, "flops": float(sweeps) * (3 * faces * 45 + 20 * n)}
    total = case["vertices"] + case["target_vertices"]
    points = case["nx"] * case["ny"]
    maps = case["steps"] * (case["runs"] + int(case["avg"]))
    flops = maps * sum(3 * _step_flops(points, k, 1) for k in range(6)) + 40962 * (300 * 200 + 2 * 7.0 * 2 * 1100)
    return {"bytes": total * (24 + 24) + 12 * case["vertices"], "flops": flops}


# ------------------------------------------------------------------ 64-bit results


def _minmax_np(v):
    return (v - v.min()) / (v.max() - v.min())


def _euler(angles):
    (ca, cb, cg), (sa, sb, sg) = np.cos(angles), np.sin(angles)
    rx = np.array([[1, 0, 0], [0, ca, -sa], [0, sa, ca]])
    ry = np.array([[cb, 0, sb], [0, 1, 0], [-sb, 0, cb]])
    rz = np.array([[cg, -sg, 0], [sg, cg, 0], [0, 0, 1]])
    return rz @ ry @ rx


def _rows(y, ny):
    y = torch.remainder(y, 2 * ny)
    return torch.where(y >= ny, 2 * ny - 1 - y, y)


def _shift(f, dx, dy):
    """f at (x + dx, y + dy): x periodic, y reflected."""

    ny = f.shape[-2]
    return torch.roll(f, -dx, dims=-1)[..., _rows(torch.arange(ny, device=f.device) + dy, ny), :]


def _corners(x, y, nx, ny):
    """Flat corner indices and fractions of the bilinear cell of zero-based (x, y)."""

    fx, fy = torch.floor(x), torch.floor(y)
    x0, y0 = fx.long(), fy.long()
    x1, y1 = torch.remainder(x0 + 1, nx), _rows(y0 + 1, ny)
    x0, y0 = torch.remainder(x0, nx), _rows(y0, ny)
    return (y0 * nx + x0, y0 * nx + x1, y1 * nx + x0, y1 * nx + x1), x - fx, y - fy


def _gather(f, index):
    """f [B, C, ny, nx] at flat indices [B, ny, nx]."""

    b, c = f.shape[:2]
    flat = index.reshape(b, 1, -1).expand(b, c, -1)
    return torch.gather(f.reshape(b, c, -1), 2, flat).reshape(b, c, *index.shape[1:])


def _blend(values, dx, dy):
    dx, dy = dx.unsqueeze(1), dy.unsqueeze(1)
    return (values[0] * (1 - dx) + values[1] * dx) * (1 - dy) + (values[2] * (1 - dx) + values[3] * dx) * dy


def _sample(f, phi):
    ny, nx = f.shape[-2:]
    index, dx, dy = _corners(phi[:, 0] - 1, phi[:, 1] - 1, nx, ny)
    return [_gather(f, i) for i in index], dx, dy


def _compose(a, ja, b, jb):
    ny, nx = a.shape[-2:]
    values, dx, dy = _sample(b, a)
    period = torch.tensor([nx, ny], dtype=a.dtype, device=a.device).view(1, 2, 1, 1)
    values = [values[0]] + [v - torch.floor((v - values[0]) / period + 0.5) * period for v in values[1:]]
    c = _blend(values, dx, dy)
    if ja is None:
        return c, None
    b00, b01, b10, b11 = _blend(*_sample(jb, a)).unbind(1)
    a0, a1, a2, a3 = ja.unbind(1)
    return c, torch.stack((b00 * a0 + b10 * a1, b01 * a0 + b11 * a1, b00 * a2 + b10 * a3, b01 * a2 + b11 * a3), 1)


def _jacobian(v, scale):
    dx = (_shift(v, 1, 0) - _shift(v, -1, 0)) * (0.5 * scale)
    dy = (_shift(v, 0, 1) - _shift(v, 0, -1)) * (0.5 * scale)
    return torch.stack((dx[:, 0] + 1, dx[:, 1], dy[:, 0], dy[:, 1] + 1), 1)


def _identity(v):
    ny, nx = v.shape[-2:]
    x = torch.arange(1, nx + 1, dtype=v.dtype, device=v.device).expand(ny, nx)
    y = torch.arange(1, ny + 1, dtype=v.dtype, device=v.device).unsqueeze(1).expand(ny, nx)
    return torch.stack((x, y)).unsqueeze(0)


def _exponential(v, k, jacobian=False):
    phi, jac = _identity(v) + v / 2.0 ** k, _jacobian(v, 1.0 / 2.0 ** k) if jacobian else None
    for _ in range(k):
        phi, jac = _compose(phi, jac, phi, jac)
    return phi, jac


def _jac_div(j, v, scale):
    d00, d10, d01, d11 = _jacobian(v, scale).unbind(1)
    det = d00 * d11 - d01 * d10
    i00, i10, i01, i11 = d11 / det, -d10 / det, -d01 / det, d00 / det
    o00, o10, o01, o11 = j.unbind(1)
    return torch.stack((o00 * i00 + o01 * i10, o10 * i00 + o11 * i10, o00 * i01 + o01 * i11, o10 * i01 + o11 * i11), 1)


def _objective(source, target, phi, jac):
    k, dx, dy = _sample(source.unsqueeze(1), phi)
    k22, k12, k21, k11 = (c[:, 0] for c in k)
    diff = (k22 * (1 - dx) + k12 * dx) * (1 - dy) + (k21 * (1 - dx) + k11 * dx) * dy - target
    ddx = (k11 - k21) * dy + (k12 - k22) * (1 - dy)
    ddy = (k11 * dx + k21 * (1 - dx)) - (k12 * dx + k22 * (1 - dx))
    gx, gy = jac[:, 0] * ddx + jac[:, 1] * ddy, jac[:, 2] * ddx + jac[:, 3] * ddy
    return (0.5 * (diff * diff).sum((1, 2)), torch.stack((gx * diff, gy * diff), 1),
            torch.stack((gx * gx, gy * gy, gx * gy), 1))


def _squaring(b, a, phi, jac, k, save):
    """k squaring steps; the last value is the slot the multigrid starts from."""

    slots, cur = [phi, phi], 0
    jacs = [jac, jac]
    for step in range(k):
        j00, j10, j01, j11 = jacs[cur].unbind(1)
        det = j00 * j11 - j01 * j10
        bx, by, a00, a11, a01 = _blend(*_sample(torch.cat((b, a), 1), slots[cur])).unbind(1)
        t1, t2, t3, t4 = a00 * j00 + a01 * j10, a01 * j00 + a11 * j10, a00 * j01 + a01 * j11, a01 * j01 + a11 * j11
        inc = torch.stack((det * (bx * j00 + by * j10), det * (bx * j01 + by * j11)), 1)
        b = b + inc
        a = a + torch.stack((det * (t1 * j00 + t2 * j10), det * (t3 * j01 + t4 * j11), det * (t1 * j01 + t2 * j11)), 1)
        slots[1 - cur] = inc
        if save or step < k - 1:
            slots[1 - cur], jacs[1 - cur] = _compose(slots[cur], jacs[cur], slots[cur], jacs[cur])
            cur = 1 - cur
    if save:
        slots[0] = slots[cur]
    return b, a, slots[cur], jacs[cur], slots[0]


def _resize(f, tnx, tny):
    def taps(count, size, wrap):
        t = (torch.arange(count, dtype=f.dtype, device=f.device) + 0.5) * size / count - 0.5
        o = torch.floor(t + 0.5)
        d = [torch.abs(o + j - t) for j in (-1, 0, 1)]
        w = [torch.where(x < 0.5, 0.75 - x * x, torch.where(x < 1.5, 0.5 * (1.5 - x) ** 2, 0 * x)) for x in d]
        return [wrap(o.long() + j) for j in (-1, 0, 1)], w

    sny, snx = f.shape[-2:]
    index, w = taps(tny, sny, lambda i: _rows(i, sny))
    f = sum(wj.unsqueeze(1) * f[..., i, :] for i, wj in zip(index, w))
    index, w = taps(tnx, snx, lambda i: torch.remainder(i, snx))
    return sum(wj * f[..., i] for i, wj in zip(index, w))


def _membrane(u, mu, sx, sy, ident):
    return ((mu * 2 * (sx * sx + sy * sy) + ident) * u - mu * sy * sy * (_shift(u, 0, -1) + _shift(u, 0, 1))
            - mu * sx * sx * (_shift(u, -1, 0) + _shift(u, 1, 0)))


def _relax(h, b, u, nit, mu, sx, sy, ident):
    ny, nx = u.shape[-2:]
    w00, near = mu * 2 * (sx * sx + sy * sy) + ident, 1.0000000001
    odd = ((torch.arange(nx, device=u.device) + torch.arange(ny, device=u.device).unsqueeze(1)) & 1).bool()
    dxx, dyy, cr = h[:, 0] + w00, h[:, 1] + w00, h[:, 2]
    det = dxx * dyy * near - cr * cr
    for it in range(2 * nit):
        r = b + mu * sy * sy * (_shift(u, 0, -1) + _shift(u, 0, 1)) + mu * sx * sx * (_shift(u, -1, 0) + _shift(u, 1, 0))
        new = torch.stack(((dyy * r[:, 0] - cr * r[:, 1]) / det, (-cr * r[:, 0] + dxx * r[:, 1]) / det), 1)
        u = torch.where(odd if it % 2 == 0 else ~odd, new, u)
    return u


def _cycle(level, hs, b, u, ps, nit):
    args = ps[level]
    u = _relax(hs[level], b, u, nit, *args)
    if level == len(hs) - 1:
        return u
    h = hs[level]
    hu = torch.stack((h[:, 0] * u[:, 0] + h[:, 2] * u[:, 1], h[:, 2] * u[:, 0] + h[:, 1] * u[:, 1]), 1)
    ny, nx = hs[level + 1].shape[-2:]
    coarse = _resize(b - _membrane(u, *args) - hu, nx, ny)
    u = u + _resize(_cycle(level + 1, hs, coarse, torch.zeros_like(coarse), ps, nit), *reversed(u.shape[-2:]))
    return _relax(h, b, u, nit, *args)


def _step(source, target, v, k, params, code=1, cycles=3, nit=3, lmreg=1e-3):
    """One membrane DARTEL step of a batch in 64 bits (the multigrid starts from the last map, never zero)."""

    s = 1.0 / 2.0 ** k
    phi, jac = _exponential(v, k, True)
    obj, rhs, hess = _objective(source, target, phi, _jac_div(jac, v, s))
    rhs, hess, phi, jac, start = _squaring(rhs, hess, _identity(v) - v * s, _jacobian(v, -s), k, code == 1)
    if code == 1:
        robj, rrhs, rhess = _objective(target, source, phi, _jac_div(jac, v, -s))
        rrhs, rhess, _, _, start = _squaring(rrhs, rhess, _identity(v) + v * s, _jacobian(v, s), k, False)
        obj, rhs, hess = obj + robj, rhs - rrhs, hess + rhess
    sx, sy, mu, _, ident = params
    reg = _membrane(v, mu, sx, sy, ident)
    rhs, hess = rhs * s + reg, hess * s
    metrics = torch.stack((obj, 0.5 * (reg * v).sum((1, 2, 3)), (rhs * rhs).sum((1, 2, 3)).sqrt()), 1)
    hs, ps, (ny, nx) = [hess], [(mu, sx, sy, ident + lmreg)], v.shape[-2:]
    while hs[-1].shape[-1] >= 2 or hs[-1].shape[-2] >= 2:
        cy, cx = ((n + 1) // 2 for n in hs[-1].shape[-2:])
        hs.append(_resize(hs[-1], cx, cy))
        ps.append((mu, sx * cx / nx, sy * cy / ny, ident + lmreg))
        if cx < 2 and cy < 2:
            break
    u = start
    for _ in range(cycles):
        u = _cycle(0, hs, rhs, u, ps, nit)
    return v - u, metrics


def _solve(source, target, loop=6, its=3):
    v = torch.zeros((source.shape[0], 2) + tuple(source.shape[1:]), dtype=source.dtype, device=source.device)
    metrics = []
    for k, params in enumerate(_default_parameters(loop)):
        for _ in range(its):
            v, m = _step(source, target, v, k, params)
            metrics.append(m)
    return v, torch.stack(metrics, 1)


def _default_parameters(loop):
    """The regulariser schedule: mu 0.125, divided by 1.25 every fourth loop."""

    return [(1.0, 1.0, 0.125 / 1.25 ** (i // 4), 0.0, 0.0) for i in range(loop)]


def _type5_sheets(stencil, surface, fwhms):
    """Type-5 curvature sheets in 64 bits from the stencil's indices and weights."""

    def norm(v):
        return v.square().sum(-1).sqrt()

    faces = stencil.faces.long()
    n = stencil.sphere_points.shape[0]
    g = (surface.double()[stencil.surface_indices.long()] * stencil.surface_weights.unsqueeze(-1)).sum(1)
    edges = torch.cat([faces[:, [i, j]] for i, j in ((0, 1), (1, 0), (1, 2), (2, 1), (2, 0), (0, 2))])
    key = torch.unique(edges[:, 0] * n + edges[:, 1])
    row, col = key // n, key % n
    mean = norm(g[faces[:, [1, 2, 0]]] - g[faces]).mean().item()

    def heat(fwhm):
        iterations = max(1, math.ceil(fwhm * fwhm * 0.541011 / (mean * mean)))
        return iterations, fwhm * 0.7355345 / math.sqrt(iterations)

    def ring(w, values):
        shape = (n,) + tuple(values.shape[1:])
        return torch.zeros(shape, dtype=values.dtype, device=values.device).index_add_(0, row, w * values[col])

    ones = torch.ones((n, 1), dtype=torch.float64, device=g.device)
    smooth, den = g, 1.0 + ring(1.0, ones) / 3.0
    for _ in range(heat(50.0)[0]):
        smooth = (smooth + ring(1.0, smooth) / 3.0) / den
    p = smooth[faces]
    fn = torch.linalg.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0])
    fn = fn / norm(fn).unsqueeze(-1)
    normals = torch.zeros_like(g)
    for c in range(3):
        a, b = p[:, (c - 1) % 3] - p[:, c], p[:, (c + 1) % 3] - p[:, c]
        angle = torch.arccos(((a * b).sum(-1) / (norm(a) * norm(b))).clamp(-1, 1))
        normals.index_add_(0, faces[:, c], fn * angle.unsqueeze(-1))
    base = ((smooth - g) * normals / norm(normals).unsqueeze(-1)).sum(-1, keepdim=True)

    def unit(v):
        return (v - v.min()) / (v.max() - v.min())

    out = []
    for fwhm in fwhms:
        iterations, sigma = heat(fwhm)
        w = torch.exp(-(g[col] - g[row]).square().sum(-1, keepdim=True) / (2 * sigma * sigma))
        values, total = base, 1.0 + ring(w, ones)
        for _ in range(iterations):
            values = (values + ring(w, values)) / total
        sheet = (unit(values[:, 0])[stencil.sheet_indices.long()] * stencil.sheet_weights).sum(-1)
        out.append(unit(sheet).reshape(stencil.ny, stencil.nx))
    return out


def exact(case, seed):
    """The 64-bit results, or None: the sweeps, stages, SOR and Nelder-Mead are sequential (minutes in plain torch),
    scoring a rotation needs a closest-triangle search per point and candidate, and a registration chains them all."""

    kind = case["kind"]
    if kind not in ("step", "solve", "many", "adjoint", "sheets"):
        return None
    state = prepare(case, seed)
    if kind == "sheets":
        return _type5_sheets(state["stencils"][0], state["surfaces"][0], _fwhms(case))
    source, target = state["source"].double(), state["target"].double()
    if kind == "step":
        v, metrics = _step(source[None], target[None], state["velocity"].double()[None], case["k"],
                           (1.0, 1.0, 0.125, 0.0, 0.0), case["code"])
        return {"velocity": v[0], "metrics": metrics[0]}
    if kind == "adjoint":
        v = state["velocity"].double().requires_grad_(True)
        phi, _ = _exponential(v, case["k"])
        diff = _blend(*_sample(source.unsqueeze(1), phi))[:, 0] - target
        energy = 0.5 * (diff * diff).sum((1, 2))
        (grad,) = torch.autograd.grad(energy.sum(), v)
        return {"energy": energy.detach(), "grad": grad}
    ny, nx = source.shape[-2:]
    v, metrics = _solve(source.reshape(-1, ny, nx), target.reshape(-1, ny, nx))
    last = v.reshape(-1, case["steps"], 2, ny, nx)[:, -1]
    flows = _exponential(last, 10)[0]
    if kind == "solve":
        return {"flow": flows[0], "metrics": metrics}
    return {"flows": flows, "metrics": metrics.reshape(case["regs"], case["steps"], -1, 3)}
