"""The workloads this library is timed on, each a call a user's program makes
through a public entry point.

* ``apply``   esf_pressure_apply: the pressure operator alone, as a caller
              that runs its own Krylov loop uses it, one product a pass.
* ``solve``   esf_pressure_solve: the solver seam, in each precision, either
              for a fixed number of iterations (tolerance 1e-30, as the
              solver benchmark sets it) or to the 1e-8 residual.
* ``static``  esf_pressure_solve_static: the allocation-free FP64 solve.
* ``batch``   esf_pressure_solve_batch: many independent systems at once.
* ``step``    one coupled step (dt = 1/240) of the rubber ball at the
              reference's shipped solver settings (tolerance 0.02, at most
              500 iterations), and the fields a program reads after it.
* ``bake``    esf_rasterize_solid: a solid's rest mass from its mesh.

Sizes are cells per axis. Inputs come from the seed alone.
"""
import ctypes as C
import math

import numpy as np
import torch

import eulersf_gb300 as E
from eulersf_gb300 import abi
from eulersf_gb300.bake import rasterize_solid
from eulersf_gb300.scene import SceneDesc, icosphere

PRECISION = {"fp64": abi.ESF_FP64, "mixed": abi.ESF_MIXED, "x64": abi.ESF_MIXED_X64}


def listed():
    return [
        # one operator product on a small grid: launch latency
        {"name": "apply_32", "kind": "apply", "nx": 32, "ny": 32, "nz": 32},
        # the operator at the benchmark's size
        {"name": "apply_256", "kind": "apply", "nx": 256, "ny": 256, "nz": 256},
        # the default precision on the low-resolution ball's grid
        {"name": "solve_fp64_64", "kind": "solve", "nx": 64, "ny": 64, "nz": 64, "precision": "fp64",
         "iters": 100, "eps": 1e-30},
        # the same on a larger box with odd sides
        {"name": "solve_fp64_ragged", "kind": "solve", "nx": 161, "ny": 127, "nz": 190, "precision": "fp64",
         "iters": 40, "eps": 1e-30},
        # a host that reserves its device memory: the allocation-free solve
        {"name": "static_48", "kind": "static", "nx": 48, "ny": 48, "nz": 48, "iters": 60, "eps": 1e-30},
        # mixed precision to the configured 1e-8 residual: several refinements
        {"name": "solve_mixed_64", "kind": "solve", "nx": 64, "ny": 64, "nz": 64, "precision": "mixed",
         "iters": 20000, "eps": 1e-8},
        # the headline's inner iteration at its size
        {"name": "solve_mixed_256", "kind": "solve", "nx": 256, "ny": 256, "nz": 256, "precision": "mixed",
         "iters": 100, "eps": 1e-30},
        # the double-float run at a serving size
        {"name": "solve_x64_160", "kind": "solve", "nx": 160, "ny": 160, "nz": 160, "precision": "x64",
         "iters": 100, "eps": 1e-30},
        # small independent systems in one call
        {"name": "batch_32x64", "kind": "batch", "nx": 32, "ny": 32, "nz": 32, "systems": 64, "iters": 100,
         "eps": 1e-30},
        # the coupled step, in each precision
        {"name": "step_fp64_64", "kind": "step", "n": 64, "precision": "fp64"},
        {"name": "step_mixed_128", "kind": "step", "n": 128, "precision": "mixed"},
        # the shipped sphere's resolution: a spacing of a hundredth of the radius
        {"name": "bake_100", "kind": "bake", "level": 3, "per_radius": 100},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["apply", "apply", "solve", "solve", "solve", "static", "batch", "step", "bake"])
    if kind == "step":
        return {"kind": kind, "n": _log_int(rng, 24, 96), "precision": rng.choice(["fp64", "mixed", "x64"])}
    if kind == "bake":
        return {"kind": kind, "level": rng.choice([2, 3]), "per_radius": _log_int(rng, 20, 80)}
    hi = {"apply": 256, "solve": 176, "static": 64, "batch": 48}[kind]
    side = [_log_int(rng, 12, hi) for _ in range(3)]
    case = {"kind": kind, "nx": side[0], "ny": side[1], "nz": side[2]}
    if kind == "apply":
        return case
    case["iters"] = _log_int(rng, 10, 100)
    case["eps"] = 1e-30
    if kind == "solve":
        case["precision"] = rng.choice(["fp64", "mixed", "mixed", "x64"])
    if kind == "batch":
        case["systems"] = rng.randint(2, 32)
    if kind == "batch" or case.get("precision") in ("mixed", "x64"):
        if rng.random() < 0.75:  # rows of a multiple of four cells, as most grids have
            case["nx"] = max(12, case["nx"] // 4 * 4)
    return case


# ------------------------------------------------------------------- inputs
def _system(case, seed, device="cuda"):
    """Node 1/m of a fluid (density 1000) with a ball (1100 more) at a seeded
    place, the Jacobi diagonal, and a right-hand side in the operator's range
    with a warm start, as consecutive steps give the solver."""
    gen = torch.Generator(device=device).manual_seed(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    X, Y, Z = nx + 1, ny + 1, nz + 1
    dh = 1.0 / max(nx, ny, nz)
    f64 = dict(dtype=torch.float64, device=device)
    centre = 0.3 + 0.4 * torch.rand(3, generator=gen, **f64)
    axis = [torch.arange(n, **f64) / max(n - 1, 1) for n in (Z, Y, X)]
    r2 = ((axis[0] - centre[0]) ** 2)[:, None, None] + ((axis[1] - centre[1]) ** 2)[None, :, None] \
        + ((axis[2] - centre[2]) ** 2)[None, None, :]
    density = 1000.0 + 1100.0 * (r2 <= 0.2 ** 2).to(torch.float64)
    minv = 1.0 / (density * dh ** 3)
    diag = _diagonal(minv)
    b = _operator(minv, torch.randn((nz, ny, nx), generator=gen, **f64))
    x0 = 0.1 * torch.randn((nz, ny, nx), generator=gen, **f64)
    return minv, diag, b, x0, dh


def _inner(minv):
    m = minv.clone()
    m[0], m[-1], m[:, 0], m[:, -1], m[:, :, 0], m[:, :, -1] = 0, 0, 0, 0, 0, 0
    return m


def _sum(a, d):
    n = a.shape[d] - 1
    return a.narrow(d, 0, n) + a.narrow(d, 1, n)


def _dif(a, d):
    n = a.shape[d] - 1
    return a.narrow(d, 0, n) - a.narrow(d, 1, n)


def _diagonal(minv):
    return 3.0 * _sum(_sum(_sum(_inner(minv), 0), 1), 2)


def _operator(minv, v):
    """J diag(1/m) J^T v, written with differences and sums along each axis."""
    m = _inner(minv)
    p = torch.nn.functional.pad(v, (1, 1, 1, 1, 1, 1))
    sz = _sum(p, 0)
    gx = _dif(_sum(sz, 1), 2) * m
    gy = _dif(_sum(sz, 2), 1) * m
    gz = _sum(_sum(_dif(p, 0), 1), 2) * m
    return -(_dif(_sum(_sum(gx, 0), 1), 2) + _dif(_sum(_sum(gy, 0), 2), 1) + _dif(_sum(_sum(gz, 1), 2), 0))


def _grid(case, dh):
    return abi.Grid(case["nx"] + 1, case["ny"] + 1, case["nz"] + 1, dh, (C.c_double * 3)(0, 0, 0))


def _mesh(case, seed):
    """A closed ball-like surface with seeded dents, 0.2 across on every axis."""
    rng = np.random.default_rng(seed)
    verts, faces = icosphere(case["level"], 0.1)
    k = rng.uniform(-12.0, 12.0, (4, 3)) / 0.1 * 0.2
    phase = rng.uniform(0.0, 2.0 * np.pi, 4)
    bump = sum(np.sin(verts @ k[i] + phase[i]) for i in range(4))
    verts = verts * (1.0 + 0.03 * bump)[:, None]
    lo, hi = verts.min(0), verts.max(0)
    return np.where(verts == hi, 0.1, -0.1 + (verts - lo) * (0.2 / (hi - lo))), faces


def _scene(case, seed):
    n = case["n"]
    return SceneDesc(N=n, eps=0.02, max_iters=500, mass_sample_dh=(1.0 / n) / 4, noise_seed=seed)


def prepare(case, seed):
    kind = case["kind"]
    lib = E.load(build_if_missing=True)
    if kind == "step":
        return {"case": case, "integrator": E.make_scene(_scene(case, seed), precision=PRECISION[case["precision"]])}
    if kind == "bake":
        verts, faces = _mesh(case, seed)
        return {"case": case, "verts": verts, "faces": faces}
    if kind == "batch":
        n = case["systems"]
        systems = [_system(case, seed * 1000 + i) for i in range(n)]
        x0 = torch.stack([s[3] for s in systems])
        x = torch.empty_like(x0)
        arr = lambda ts: (C.c_void_p * n)(*[t.data_ptr() for t in ts])
        return {"case": case, "lib": lib, "systems": systems, "x0": x0, "x": x,
                "grids": (abi.Grid * n)(*[_grid(case, s[4]) for s in systems]),
                "m": arr([s[0] for s in systems]), "d": arr([s[1] for s in systems]),
                "b": arr([s[2] for s in systems]), "xs": arr(x.unbind(0))}
    minv, diag, b, x0, dh = _system(case, seed)
    state = {"case": case, "lib": lib, "grid": _grid(case, dh), "minv": minv}
    if kind == "apply":
        return dict(state, v=x0, out=torch.empty_like(x0))
    return dict(state, diag=diag, b=b, x0=x0, x=torch.empty_like(x0))


# --------------------------------------------------------------------- pass
def _ptr(t):
    return C.c_void_p(t.data_ptr())


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _check(status, what):
    if status != 0:
        raise abi.EsfError(status, what, E.last_error())


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "step":
        scene = state["integrator"]
        report = scene.stepImplicit()
        return {"velocity": scene.get("velocity"), "pressure": scene.get("lambda1"),
                "mesh": scene.get("solid.meshVertices"),
                "iterations": report["iterations"]}
    if kind == "bake":
        res, dh, origin, mass, total = rasterize_solid(state["verts"], state["faces"],
                                                       0.1 / case["per_radius"], 1000.0)
        return {"mass": mass, "total": np.float64(total), "res": list(res)}
    lib = state["lib"]
    if kind == "apply":
        _check(lib.esf_pressure_apply(C.byref(state["grid"]), _ptr(state["minv"]), _ptr(state["v"]),
                                      _ptr(state["out"]), _stream()), "esf_pressure_apply")
        return state["out"]
    state["x"].copy_(state["x0"])  # the warm start a step begins from
    if kind == "batch":
        n = case["systems"]
        its, rel = (C.c_int * n)(), (C.c_double * n)()
        _check(lib.esf_pressure_solve_batch(n, state["grids"], state["m"], state["d"], state["b"], state["xs"],
                                            case["eps"], case["iters"], abi.ESF_MIXED, 0, its, rel, None,
                                            _stream()), "esf_pressure_solve_batch")
        return {"x": state["x"], "iterations": np.array(its)}
    its, rel = C.c_int(), C.c_double()
    system = (C.byref(state["grid"]), _ptr(state["minv"]), _ptr(state["diag"]), _ptr(state["b"]),
              _ptr(state["x"]), case["eps"], case["iters"])
    if kind == "static":
        _check(lib.esf_pressure_solve_static(*system, C.byref(its), C.byref(rel), _stream()),
               "esf_pressure_solve_static")
    else:
        _check(lib.esf_pressure_solve(*system, PRECISION[case["precision"]], C.byref(its), C.byref(rel),
                                      _stream()), "esf_pressure_solve")
    return {"x": state["x"], "iterations": its.value}


# ------------------------------------------------------------- what it takes
# Words a row and iteration of the conjugate residual method moves when each
# vector is read and written once: r, t, q, d and x in and out, 1/diag and 1/m
# in; and the arithmetic of one operator product with the vector updates.
ITERATION_WORDS, ITERATION_FLOPS, PRODUCT_FLOPS = 12, 54, 36
STEP_WORDS = 60  # node fields the step reads and writes once each (FP64)


def work(case):
    kind = case["kind"]
    if kind == "step":
        nodes = (case["n"] + 1) ** 3
        return {"bytes": STEP_WORDS * 8 * nodes, "flops": 400 * nodes}
    if kind == "bake":
        nodes = (2.0 * case["per_radius"] + 20) ** 3
        return {"bytes": 8 * nodes, "flops": 0}
    rows = case["nx"] * case["ny"] * case["nz"]
    nodes = (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1)
    if kind == "apply":
        return {"bytes": 8 * (2 * rows + nodes), "flops": PRODUCT_FLOPS * rows}
    mixed = kind == "batch" or case.get("precision", "fp64") != "fp64"
    word = 4 if mixed else 8
    words = ITERATION_WORDS + (4 if case.get("precision") == "x64" else 0)
    iters = min(case["iters"], 500)  # to the 1e-8 residual: some hundreds at the least
    one = 8 * (4 * rows + nodes) + iters * words * word * rows
    n = case.get("systems", 1)
    return {"bytes": n * one, "flops": n * iters * ITERATION_FLOPS * rows}


# ------------------------------------------------------------- 64-bit values
def _residual_method(minv, diag, b, x, iters, inner_eps):
    """x after `iters` iterations of the Jacobi-preconditioned conjugate
    residual method; with `inner_eps` the mixed solve's scheme, which starts
    anew from the true residual whenever r.Ar has fallen by inner_eps^2."""
    done = 0
    while done < iters:
        r = (b - _operator(minv, x)) / diag
        s = _operator(minv, r)
        delta = delta0 = float((r * s).sum())
        d, ad, beta = torch.zeros_like(r), torch.zeros_like(r), 0.0
        while done < iters:
            d = beta * d + r
            ad = beta * ad + s
            q = ad / diag
            alpha = delta / float((ad * q).sum())
            x = x + alpha * d
            r = r - alpha * q
            s = _operator(minv, r)
            new = float((r * s).sum())
            beta, delta = new / delta, new
            done += 1
            if inner_eps and delta <= inner_eps ** 2 * delta0:
                break
    return x


def _bake_mass(case, seed):
    verts, faces = _mesh(case, seed)
    dh = 0.1 / case["per_radius"]
    lo, hi = verts.min(0) - dh * 10, verts.max(0) + dh * 10
    res = [int(v) for v in (hi - lo) / dh]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f64 = dict(dtype=torch.float64, device=dev)
    tri = torch.tensor(verts[faces], **f64)  # (n, 3, 3)
    low = torch.tensor(lo, **f64)
    a, b, c = tri[None, :, 0], tri[None, :, 1], tri[None, :, 2]
    normal = torch.linalg.cross(b - a, c - a)
    normal = normal / normal.norm(dim=-1, keepdim=True)
    total = res[0] * res[1] * res[2]
    solid = torch.empty(total, dtype=torch.bool, device=dev)
    step = max(1, 1 << 22 >> max(1, len(faces)).bit_length() - 1)
    for n0 in range(0, total, step):
        n = torch.arange(n0, min(total, n0 + step), device=dev)
        p = torch.stack([n % res[0], n // res[0] % res[1], n // (res[0] * res[1])], -1).to(torch.float64) * dh + low
        p = p[:, None]
        best, over = None, None
        for u, v in ((a, b), (b, c), (c, a)):
            e, w = v - u, p - u
            t = ((w * e).sum(-1) / (e * e).sum(-1)).clamp(0, 1)
            d2 = (w - t[..., None] * e).square().sum(-1)
            best = d2 if best is None else torch.minimum(best, d2)
            side = (torch.linalg.cross(normal, e.expand_as(normal)) * w).sum(-1) >= 0
            over = side if over is None else over & side
        plane = ((p - a) * normal).sum(-1).square()
        best = torch.where(over, torch.minimum(best, plane), best).amin(1)
        x, y, z = a - p, b - p, c - p
        lx, ly, lz = x.norm(dim=-1), y.norm(dim=-1), z.norm(dim=-1)
        det = (x * torch.linalg.cross(y, z)).sum(-1)
        den = lx * ly * lz + (x * y).sum(-1) * lz + (y * z).sum(-1) * lx + (z * x).sum(-1) * ly
        angle = 2.0 * torch.atan2(det, den).sum(1)
        dist = best.sqrt()
        solid[n0:n0 + step] = torch.where(angle.abs() > 2.0 * math.pi, -dist, dist) <= 0.5 * dh
    mass = solid.to(torch.float64) * 1000.0
    return {"mass": mass.reshape(res[2], res[1], res[0]), "total": mass.sum() * dh ** 3, "res": None}


def exact(case, seed):
    kind = case["kind"]
    if kind == "step":  # a whole engine: no 64-bit value apart from its own
        return None
    if kind == "bake":
        return _bake_mass(case, seed)
    if kind == "batch":
        xs = []
        for i in range(case["systems"]):
            minv, diag, b, x0, dh = _system(case, seed * 1000 + i)
            xs.append(_residual_method(minv, diag, b, x0, case["iters"], 1e-4))
        return {"x": torch.stack(xs), "iterations": None}
    if kind == "solve" and (case["eps"] > 1e-20 or case["precision"] == "x64"):
        return None  # stops (or replaces its residual) where its own rounding says
    minv, diag, b, x0, dh = _system(case, seed)
    if kind == "apply":
        return _operator(minv, x0)
    inner = 1e-4 if case.get("precision", "fp64") == "mixed" else None
    return {"x": _residual_method(minv, diag, b, x0, case["iters"], inner), "iterations": None}
