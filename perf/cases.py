"""The measured cases: the work a user of toptimization_b200 has it do.

A topology optimisation is a few hundred OC iterations; nearly all of the time
goes into the PCG solves, the rest into the density filter, the sensitivities,
the dc filter and the OC update. The cases are those parts, each through the
entry point a program calls (`PCGSolver.solve`, `kernels.matvec`, the filters,
`kernels.sensitivity`, `oc_update`), and whole runs (`simp.run`, `Batch`):

  run_mbb_60x20           the smallest configuration (examples/mbb_60x20.yaml):
                          a whole run, where launches and latency count
  run_cantilever_400x200  the middle configuration through the CUDA-graph
                          engine, nodal block-Jacobi
  solve_bridge_mixed      the largest configuration's solve, mixed precision
  solve_bridge_fp64       the same in plain FP64
  solve_ragged_block      the reference's element-block preconditioner, an odd grid
  solve_small_jacobi      one solve of a small odd grid (first design studies)
  solve_solid_jacobi      the 3D configuration's solve (128x64x64)
  solve_solid_block       3D with the element-block preconditioner, an odd grid
  design_bridge           all of an OC iteration but its solve, 2048x1024
  design_ragged_sens      the same with the sensitivity filter, an odd middle grid
  design_solid            the same in 3D
  batch_uneven            uneven designs advanced together (the batched engine)

`draw` gives more of the same kinds (and `matvec`, a stiffness application on
its own, FP64 and FP32), sizes spread over the whole range. Solves are capped
at a number of PCG iterations, so that a pass is the same work for every seed;
a run's real solves take hundreds (60x20) to ten thousand (2048x1024). Mixed
solves start a run (uniform density, u = 0): after some tens of iterations on a
contrasty density two FP32-stored Krylov sequences that differ in one rounding
are no longer comparable, whatever computes them. The element-block solves, as
sensitive in FP64 on such a density, take the grey one of a run's first iterations.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from toptimization_b200 import _lib
from toptimization_b200.batch import Batch
from toptimization_b200.fem import kernels
from toptimization_b200.fem.solver import PCGSolver
from toptimization_b200.material import compute_Ke_2d, compute_Ke_3d, regularized_inverse
from toptimization_b200.mesh import fixed_node_mask, force_vector
from toptimization_b200.optimizer import filter as filt
from toptimization_b200.optimizer import oc
from toptimization_b200.optimizer.simp import RunHistory, run as simp_run
from toptimization_b200.problem import problem_from_dict

E_MIN, PENALTY, MOVE = 1e-9, 3.0, 0.2


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest configuration as a user runs it: a few OC iterations
        {"name": "run_mbb_60x20", "kind": "run", "nx": 60, "ny": 20, "nz": 0, "family": "mbb",
         "pre": "jacobi", "precision": "fp64", "engine": "direct", "filter": "density",
         "rmin": 1.5, "oc": 5, "cg": 120},
        # the middle configuration, each OC iteration one CUDA graph
        {"name": "run_cantilever_400x200", "kind": "run", "nx": 400, "ny": 200, "nz": 0,
         "family": "cantilever", "pre": "nodal_block_jacobi", "precision": "fp64",
         "engine": "graph", "filter": "density", "rmin": 3.0, "oc": 4, "cg": 160},
        # the headline configuration's solve, both precisions: the run's first
        # solve (uniform density) in the mixed form, a mid-run density in FP64
        {"name": "solve_bridge_mixed", "kind": "solve", "nx": 2048, "ny": 1024, "nz": 0,
         "family": "bridge", "pre": "nodal_block_jacobi", "precision": "mixed", "cg": 48},
        {"name": "solve_bridge_fp64", "kind": "solve", "nx": 2048, "ny": 1024, "nz": 0,
         "family": "bridge", "pre": "nodal_block_jacobi", "precision": "fp64", "cg": 64},
        # the reference's element-block preconditioner on a grid of odd sizes
        {"name": "solve_ragged_block", "kind": "solve", "nx": 801, "ny": 395, "nz": 0,
         "family": "cantilever", "pre": "block_jacobi", "precision": "fp64", "cg": 40},
        # a small study: latency of the iteration
        {"name": "solve_small_jacobi", "kind": "solve", "nx": 151, "ny": 49, "nz": 0,
         "family": "mbb", "pre": "jacobi", "precision": "fp64", "cg": 100},
        # 3D: the configuration, and an odd grid with the element-block preconditioner
        {"name": "solve_solid_jacobi", "kind": "solve", "nx": 128, "ny": 64, "nz": 64,
         "family": "cantilever", "pre": "jacobi", "precision": "fp64", "cg": 64},
        {"name": "solve_solid_block", "kind": "solve", "nx": 61, "ny": 31, "nz": 29,
         "family": "cantilever", "pre": "block_jacobi", "precision": "fp64", "cg": 40},
        # an OC iteration without its solve: filter, sensitivity, dc filter, OC update
        {"name": "design_bridge", "kind": "design", "nx": 2048, "ny": 1024, "nz": 0,
         "filter": "density", "rmin": 4.0},
        {"name": "design_ragged_sens", "kind": "design", "nx": 517, "ny": 173, "nz": 0,
         "filter": "sensitivity", "rmin": 2.5},
        {"name": "design_solid", "kind": "design", "nx": 128, "ny": 64, "nz": 64,
         "filter": "density", "rmin": 1.5},
        # uneven designs together (nelx 64..512, aspect 1..3, the batch workload's families)
        {"name": "batch_uneven", "kind": "batch", "designs": 16, "mix": 1, "lo": 64, "hi": 512,
         "oc": 2, "cg": 40},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve3", "design", "design3", "run", "matvec", "batch"])
    nx = _log_int(rng, 32, 2048)
    ny = max(8, min(1024, int(nx / rng.uniform(1.0, 3.0))))
    n3 = [_log_int(rng, 8, 128), _log_int(rng, 6, 64), _log_int(rng, 6, 64)]
    if kind == "solve":
        pre = rng.choice(["jacobi", "nodal_block_jacobi", "none", "block_jacobi"])
        precision = rng.choice(["fp64", "mixed"]) if pre in ("jacobi", "nodal_block_jacobi") \
            else "fp64"
        return {"kind": "solve", "nx": nx, "ny": ny, "nz": 0,
                "family": rng.choice(["mbb", "cantilever", "bridge"]), "pre": pre,
                "precision": precision,
                "cg": rng.randrange(16, 25) if pre == "block_jacobi" else rng.randrange(24, 49)}
    if kind == "solve3":
        pre = rng.choice(["jacobi", "jacobi", "block_jacobi", "none"])
        return {"kind": "solve", "nx": n3[0], "ny": n3[1], "nz": n3[2], "family": "cantilever",
                "pre": pre, "precision": "fp64",
                "cg": rng.randrange(16, 25) if pre == "block_jacobi" else rng.randrange(24, 49)}
    if kind == "design":
        return {"kind": "design", "nx": nx, "ny": ny, "nz": 0,
                "filter": rng.choice(["density", "density", "sensitivity"]),
                "rmin": round(rng.uniform(1.2, 6.0), 2)}
    if kind == "design3":
        return {"kind": "design", "nx": n3[0], "ny": n3[1], "nz": n3[2],
                "filter": rng.choice(["density", "density", "sensitivity"]),
                "rmin": round(rng.uniform(1.2, 3.2), 2)}
    if kind == "matvec":
        return {"kind": "matvec", "nx": nx, "ny": ny, "nz": 0,
                "dtype": rng.choice(["float64", "float32"])}
    if kind == "batch":
        hi = _log_int(rng, 96, 512)
        return {"kind": "batch", "designs": rng.randrange(3, 17), "mix": rng.randrange(1 << 20),
                "lo": max(32, hi // 4), "hi": hi, "oc": 2, "cg": rng.randrange(16, 41)}
    nx = _log_int(rng, 32, 400)
    return {"kind": "run", "nx": nx, "ny": max(8, int(nx / rng.uniform(1.0, 3.0))), "nz": 0,
            "family": rng.choice(["mbb", "cantilever", "bridge"]),
            "pre": rng.choice(["jacobi", "nodal_block_jacobi"]), "precision": "fp64",
            "engine": rng.choice(["direct", "graph"]),
            "filter": rng.choice(["density", "density", "sensitivity"]),
            "rmin": round(rng.uniform(1.5, 4.0), 2), "oc": rng.randrange(2, 5),
            "cg": rng.randrange(40, 81)}


# ---------------------------------------------------------------- inputs
def _problem(c, frac, volfrac, rmin=1.5, max_iter=1, max_cg=100):
    """The configuration's YAML mapping: an MBB half-beam, a cantilever or a
    bridge, with the load at fraction `frac` of the loaded edge (the bridge:
    spread over the whole deck)."""
    nx, ny, nz, family = c["nx"], c["ny"], c["nz"], c["family"]
    if nz:
        iy = int(round(frac * ny))
        fixed = [{"nodes": {"type": "face", "face": "left"}, "dofs": ["x", "y", "z"]}]
        loads = [{"nodes": {"type": "region", "x": [nx, nx], "y": [iy, iy], "z": [0, nz]},
                  "force": [0.0, -1.0 / (nz + 1), 0.0]}]
    elif family == "mbb":
        fixed = [{"nodes": {"type": "edge", "edge": "left"}, "dofs": ["x"]},
                 {"nodes": {"type": "point", "location": [nx, 0]}, "dofs": ["y"]}]
        loads = [{"nodes": {"type": "point", "location": [int(round(frac * nx)), ny]},
                  "force": [0.0, -1.0]}]
    elif family == "cantilever":
        fixed = [{"nodes": {"type": "edge", "edge": "left"}, "dofs": ["x", "y"]}]
        loads = [{"nodes": {"type": "point", "location": [nx, int(round(frac * ny))]},
                  "force": [0.0, -1.0]}]
    else:
        fixed = [{"nodes": {"type": "point", "location": [x, 0]}, "dofs": ["x", "y"]}
                 for x in (0, nx)]
        if family == "bridge":
            loads = [{"nodes": {"type": "edge", "edge": "top"}, "force": [0.0, -1.0 / (nx + 1)]}]
        else:  # the uneven-design workload's bridge: one load on the deck
            loads = [{"nodes": {"type": "point", "location": [int(round(frac * nx)), ny]},
                      "force": [0.0, -1.0]}]
    return problem_from_dict({
        "problem": {"name": family, "dimension": 3 if nz else 2},
        "domain": {"nelx": nx, "nely": ny, **({"nelz": nz} if nz else {})},
        "material": {"E": 1.0, "nu": 0.3, "E_min": E_MIN},
        "boundary_conditions": {"fixed": fixed}, "loads": loads,
        "optimization": {"volume_fraction": volfrac, "penalty": PENALTY, "filter_radius": rmin,
                         "filter_type": c.get("filter", "density"), "max_iterations": max_iter,
                         "tolerance": 0.0, "move_limit": MOVE},
        "solver": {"max_cg_iterations": max_cg, "cg_tolerance": 1e-8,
                   "preconditioner": c.get("pre", "nodal_block_jacobi"),
                   "precision": c.get("precision", "fp64"), "inner_tolerance": 1e-3,
                   "max_outer_iterations": 50},
        "output": {"directory": "results/cases"}})


def _axes(c, device, centre):
    n = [c["nx"], c["ny"]] + ([c["nz"]] if c["nz"] else [])
    off = 0.5 if centre else 0.0
    ax = [(torch.arange(k + (0 if centre else 1), dtype=torch.float64, device=device) + off) / k
          for k in n]
    return torch.meshgrid(*ax, indexing="ij")


def _density(c, rng, device):
    """A mid-run physical density: bars of material with soft edges, voids at
    the lower bound, and solid where a load or a support may sit (the boundary)."""
    X = _axes(c, device, True)
    field = torch.zeros_like(X[0])
    for _ in range(6):
        k, ph = rng.uniform(1.0, 6.0, len(X)), rng.uniform(0.0, 6.28)
        field += rng.uniform(0.5, 1.0) * torch.cos(sum(float(a) * 3.14159 * x
                                                       for a, x in zip(k, X)) + float(ph))
    rho = torch.sigmoid(3.0 * field)
    n = [c["nx"], c["ny"]] + ([c["nz"]] if c["nz"] else [])
    for d, (x, k) in enumerate(zip(X, n)):
        rim = torch.minimum(x, 1.0 - x) * k < 3.0
        if d < 2:
            rho = torch.where(rim, torch.clamp(rho, min=0.9), rho)
    return torch.clamp(rho, 0.001, 1.0).reshape(-1).contiguous()


def _displacement(c, rng, device):
    """A bending displacement with some local waviness, scaled like a unit load's."""
    X = _axes(c, device, False)
    comps = []
    for d in range(len(X)):
        v = torch.zeros_like(X[0])
        for _ in range(4):
            k, ph = rng.uniform(0.5, 9.0, len(X)), rng.uniform(0.0, 6.28)
            v += rng.uniform(-1.0, 1.0) * torch.sin(sum(float(a) * x for a, x in zip(k, X))
                                                    + float(ph)) * X[0] ** 2
        comps.append(30.0 * v)
    return torch.stack([v.reshape(-1) for v in comps], dim=1).reshape(-1).contiguous()


def _grid(c):
    if c["nz"]:
        return _lib.grid3(c["nx"], c["ny"], c["nz"], E_MIN, PENALTY)
    return _lib.grid(c["nx"], c["ny"], E_MIN, PENALTY)


def _stiffness(nz):
    Ke = compute_Ke_3d(1.0, 0.3) if nz else compute_Ke_2d(1.0, 0.3)
    inv, alpha = regularized_inverse(Ke)
    (_lib.ensure_stiffness3 if nz else _lib.ensure_stiffness)(Ke, inv, alpha)


def _run_problem(c, rng):
    return _problem(c, float(rng.uniform(0.1, 0.9)), float(rng.uniform(0.3, 0.6)), c["rmin"],
                    c["oc"], c["cg"])


def _batch_problems(c, rng):
    """Sizes and families come from the case's mix, loads and volumes from the seed."""
    mix, out = np.random.default_rng(c["mix"]), []
    for _ in range(c["designs"]):
        nx = int(mix.integers(c["lo"], c["hi"] + 1))
        d = {"nx": nx, "ny": max(8, int(round(nx / int(mix.integers(1, 4))))), "nz": 0,
             "family": ["mbb", "cantilever", "bridge_point"][int(mix.integers(0, 3))],
             "precision": "mixed"}
        out.append(_problem(d, float(rng.uniform(0.1, 0.9)), float(rng.uniform(0.3, 0.6)),
                            float(rng.uniform(1.5, 4.0)), c["oc"], c["cg"]))
    return out


def _solve_inputs(c, seed, device):
    rng = np.random.default_rng(seed)
    pr = _problem(c, float(rng.uniform(0.2, 0.8)), 0.4, 1.5, 1, c["cg"])
    f = force_vector(pr)
    if c["precision"] == "mixed":
        rho = torch.full((c["nx"] * c["ny"],), float(rng.uniform(0.3, 0.6)), dtype=torch.float64,
                         device=device)
    else:
        rho = _density(c, rng, device)
        if c["pre"] == "block_jacobi":
            rho = 0.4 * (0.5 + rho)
    return {"f": torch.from_numpy(f).to(device), "f2": float(np.dot(f, f)),
            "fixed": torch.from_numpy(fixed_node_mask(pr)).to(device), "rho": rho}


def _design_inputs(c, seed, device):
    rng = np.random.default_rng(seed)
    return {"rho": _density(c, rng, device), "u": _displacement(c, rng, device)}


def _matvec_inputs(c, seed, device):
    rng = np.random.default_rng(seed)
    dtype = getattr(torch, c["dtype"])
    pr = _problem(dict(c, family="cantilever"), 0.5, 0.4)
    gen = torch.Generator(device=device).manual_seed(int(seed))
    p = torch.randn(2 * (c["nx"] + 1) * (c["ny"] + 1), generator=gen, device=device,
                    dtype=torch.float64)
    return {"rho": _density(c, rng, device).to(dtype), "p": p.to(dtype),
            "fixed": torch.from_numpy(fixed_node_mask(pr)).to(device)}


def prepare(case, seed):
    c, dev = case, torch.device("cuda", torch.cuda.current_device())
    kind = c["kind"]
    if kind == "run":
        return {"c": c, "problem": _run_problem(c, np.random.default_rng(seed))}
    if kind == "batch":
        _stiffness(0)
        return {"c": c, "problems": _batch_problems(c, np.random.default_rng(seed))}
    _stiffness(c["nz"])
    if kind == "solve":
        s = _solve_inputs(c, seed, dev)
        s["solver"] = PCGSolver(c["nx"], c["ny"], E_MIN, PENALTY, s["f2"],
                                preconditioner=c["pre"], precision=c["precision"],
                                max_iter=c["cg"], tol=1e-8, nelz=c["nz"], device=dev)
        s["u"] = torch.zeros_like(s["f"])
    elif kind == "design":
        s = _design_inputs(c, seed, dev)
        g = s["grid"] = _grid(c)
        s["volfrac"] = float(s["rho"].mean())
        for k in ("phys", "dc", "dcf", "new"):
            s[k] = torch.empty_like(s["rho"])
        s["scalars"] = torch.zeros(5, dtype=torch.float64, device=dev)
        s["sens_ws"] = kernels.sensitivity_workspace(g, dev)
        s["oc_ws"] = oc.oc_workspace(g, dev)
    else:
        s = _matvec_inputs(c, seed, dev)
        s["grid"] = _grid(c)
        s["ap"] = torch.empty_like(s["p"])
        s["ws"] = kernels.matvec_workspace(s["grid"], dev)
    s["c"] = c
    return s


# ---------------------------------------------------------------- one pass
def run(s):
    c = s["c"]
    kind = c["kind"]
    if kind == "run":
        hist = RunHistory()
        rho = simp_run(s["problem"], live_viz=False, verbose=False, save=False, history=hist,
                       engine=c["engine"])
        return {"density": rho, "compliance": np.array(hist.compliance),
                "volume": np.array(hist.volume)}
    if kind == "batch":
        b = Batch(c["designs"])
        slots = [b.add(p) for p in s["problems"]]
        b.run()
        out = [b.density(k).reshape(-1) for k in slots]
        comp = np.concatenate([b.history(k)["compliance"] for k in slots])
        b.close()
        return {"density": np.concatenate(out), "compliance": comp}
    if kind == "solve":
        info = s["solver"].solve(s["rho"], s["f"], s["fixed"], s["u"], warm_start=False)
        return {"u": s["u"], "iters": int(info.iters)}
    if kind == "design":
        g, sc = s["grid"], s["scalars"]
        if c["filter"] == "density":
            filt.density_filter(g, c["rmin"], s["rho"], s["phys"])
            kernels.sensitivity(g, s["phys"], s["u"], s["dc"], sc[0:1], s["sens_ws"])
            filt.density_filter(g, c["rmin"], s["dc"], s["dcf"])
        else:
            kernels.sensitivity(g, s["rho"], s["u"], s["dc"], sc[0:1], s["sens_ws"])
            filt.sensitivity_filter(g, c["rmin"], s["rho"], s["dc"], s["dcf"])
        oc.oc_update(g, s["volfrac"], MOVE, s["rho"], s["dcf"], s["new"], sc[1:5], s["oc_ws"])
        out = {"dc": s["dc"], "dcf": s["dcf"], "new": s["new"], "scalars": sc}
        if c["filter"] == "density":
            out["phys"] = s["phys"]
        return out
    ap, pap = kernels.matvec(s["grid"], s["rho"], s["fixed"], s["p"], s["ap"], s["ws"],
                             with_dot=True)
    return {"ap": ap, "pap": pap}


# ---------------------------------------------------------------- what it cannot do without
def _sizes(c):
    if c["nz"]:
        return (c["nx"] * c["ny"] * c["nz"], (c["nx"] + 1) * (c["ny"] + 1) * (c["nz"] + 1), 3)
    return c["nx"] * c["ny"], (c["nx"] + 1) * (c["ny"] + 1), 2


def _solve_work(c):
    """Per PCG iteration: the vectors r, p, K p and u once in and once out
    (the mixed form's Krylov vectors in 4 bytes), the element scales and mask."""
    E, N, d = _sizes(c)
    v = 4 if c.get("precision") == "mixed" else 8
    per_b = 2 * (3 * d * N * v + d * N * 8) + E * v + N
    per_f = E * (191 if d == 3 else 40) + 14 * d * N
    k = c["cg"]
    return k * per_b + 4 * d * N * 8, k * per_f


def _design_work(c):
    E, N, d = _sizes(c)
    b = E * 8 * (2 + 3 + 2 + 3) + d * N * 8
    R = math.ceil(c["rmin"])
    taps = sum(1 for k in np.ndindex(*([2 * R + 1] * d))
               if math.dist(k, [R] * d) < c["rmin"])
    return b, E * (2 * 2 * taps + (600 if d == 3 else 80) + 40 * 6)


def work(case):
    c = case
    if c["kind"] == "solve":
        b, f = _solve_work(c)
    elif c["kind"] == "design":
        b, f = _design_work(c)
    elif c["kind"] == "matvec":
        E, N, d = _sizes(c)
        s = 8 if c["dtype"] == "float64" else 4
        b, f = 2 * d * N * s + E * s + N, 45 * E
    elif c["kind"] == "run":
        (b, f), (b2, f2) = _solve_work(c), _design_work(c)
        b, f = c["oc"] * (b + b2), c["oc"] * (f + f2)
    else:
        n = (c["lo"] + c["hi"]) / 2.0
        one = dict(c, nx=int(n), ny=int(n / 2), nz=0, precision="mixed", rmin=2.75)
        (b, f), (b2, f2) = _solve_work(one), _design_work(one)
        b, f = c["designs"] * c["oc"] * (b + b2), c["designs"] * c["oc"] * (f + f2)
    return {"bytes": float(b), "flops": float(f)}


# ---------------------------------------------------------------- the same in plain 64 bits
def _corner_bits(d):
    """Corner offsets in the element's local order (counter-clockwise, then the top face)."""
    flat = [(0, 0), (1, 0), (1, 1), (0, 1)]
    return flat if d == 2 else [(a, b, z) for z in (0, 1) for a, b in flat]


def _corner(v, off, n):
    """The nodal field v (nodes..., comps) seen at one corner of every element."""
    return v[tuple(slice(o, o + k) for o, k in zip(off, n))]


def _apply(Ke, scale, v, n):
    """K v by elements: v is shaped (nodes..., comps), scale (elements...)."""
    d = len(n)
    offs = _corner_bits(d)
    q = torch.cat([_corner(v, o, n) for o in offs], dim=-1)
    f = scale.unsqueeze(-1) * (q @ Ke.T)
    out = torch.zeros_like(v)
    for i, o in enumerate(offs):
        _corner(out, o, n).add_(f[..., d * i:d * i + d])
    return out


def _fixed_bits(mask, shape):
    return torch.stack([(mask >> k) & 1 for k in range(shape[-1])], dim=-1).reshape(shape).bool()


def _exact_pcg(n, Ke, Kinv, alpha_reg, scale, f, fixed, u, pre, iters, tol):
    """The reference's preconditioned CG, `iters` steps at most."""
    d = len(n)

    def K(v):
        y = _apply(Ke, scale, v, n)
        return torch.where(fixed, v, y)

    if pre in ("jacobi", "nodal_block_jacobi"):
        B = f.new_zeros(f.shape + (d,))
        for i, o in enumerate(_corner_bits(d)):
            blk = Ke[d * i:d * i + d, d * i:d * i + d]
            _corner(B, o, n).add_(scale[..., None, None] * blk)
        diag = torch.diagonal(B, dim1=-2, dim2=-1).clone()
        diag = torch.where(fixed, torch.ones_like(diag), torch.clamp(diag, min=1e-20))
    if pre == "nodal_block_jacobi":
        eye = torch.eye(d, dtype=f.dtype, device=f.device)
        out = fixed.unsqueeze(-1) | fixed.unsqueeze(-2)
        B = torch.where(out, eye.expand_as(B), B)
        det = B[..., 0, 0] * B[..., 1, 1] - B[..., 0, 1] * B[..., 1, 0]
    if pre == "block_jacobi":
        w = scale / torch.clamp(scale, min=alpha_reg) ** 2
        cnt = torch.zeros_like(f[..., :1])
        for o in _corner_bits(d):
            _corner(cnt, o, n).add_(1.0)
        root = torch.rsqrt(cnt)

    def M(r):
        if pre == "none":
            return r
        if pre == "jacobi":
            return r / diag
        if pre == "nodal_block_jacobi":
            x = (B[..., 1, 1] * r[..., 0] - B[..., 0, 1] * r[..., 1]) / det
            y = (B[..., 0, 0] * r[..., 1] - B[..., 1, 0] * r[..., 0]) / det
            return torch.stack([x, y], dim=-1)
        z = _apply(Kinv, w, r * root, n) * root
        return torch.where(fixed, torch.zeros_like(z), z)

    tol2 = tol * tol * float((f * f).sum())
    r = f - K(u)
    z = M(r)
    p, rz, it = z, float((r * z).sum()), 0
    for it in range(1, iters + 1):
        ap = K(p)
        alpha = rz / float((p * ap).sum())
        u = u + alpha * p
        r = r - alpha * ap
        if float((r * r).sum()) < tol2:
            break
        z = M(r)
        new = float((r * z).sum())
        p = z + (new / (rz + 1e-60)) * p
        rz = new
    return u, it


def _exact_filter(n, rmin, x):
    """sum_j w x_j and sum_j w over the hat of radius rmin."""
    R = math.ceil(rmin)
    num, den = torch.zeros_like(x), torch.zeros_like(x)
    one = torch.ones_like(x)
    for k in np.ndindex(*([2 * R + 1] * len(n))):
        off = [a - R for a in k]
        w = rmin - math.sqrt(sum(o * o for o in off))
        if w <= 0 or any(abs(o) >= m for o, m in zip(off, n)):
            continue
        to = tuple(slice(max(0, -o), m - max(0, o)) for o, m in zip(off, n))
        fr = tuple(slice(max(0, o), m - max(0, -o)) for o, m in zip(off, n))
        num[to] += w * x[fr]
        den[to] += w * one[fr]
    return num, den


def _exact_sens(n, Ke, rho, u):
    d = len(n)
    q = torch.cat([_corner(u, o, n) for o in _corner_bits(d)], dim=-1)
    uku = ((q @ Ke.T) * q).sum(-1)
    dc = -PENALTY * rho ** (PENALTY - 1) * (1.0 - E_MIN) * uku
    return dc, ((E_MIN + rho ** PENALTY * (1.0 - E_MIN)) * uku).sum()


def _exact_oc(volfrac, rho, dc):
    lo, hi, steps = 0.0, 1e9, 0
    lower, upper = torch.clamp(rho - MOVE, min=0.001), torch.clamp(rho + MOVE, max=1.0)
    while True:
        lam = 0.5 * (lo + hi)
        be = torch.clamp(-dc / (lam + 1e-20), min=0.0)
        new = torch.maximum(lower, torch.minimum(upper, rho * be.sqrt()))
        vol = float(new.mean())
        steps += 1
        if vol > volfrac:
            lo = lam
        else:
            hi = lam
        if (hi - lo) / (hi + lo + 1e-30) < 1e-4 or steps >= 50:
            break
    return new, float((new - rho).abs().max()), vol, lam, steps


def _exact_design(n, Ke, rmin, mode, rho, u, volfrac):
    """The part of an OC iteration after the solve (and before it: the filter)."""
    if mode == "density":
        num, den = _exact_filter(n, rmin, rho)
        phys = num / (den + 1e-20)
    else:
        phys = rho
    dc, comp = _exact_sens(n, Ke, phys, u)
    if mode == "density":
        num, den = _exact_filter(n, rmin, dc)
        dcf = num / (den + 1e-20)
    else:
        num, den = _exact_filter(n, rmin, rho * dc)
        dcf = num / (rho * den + 1e-20)
    new, chg, vol, lam, steps = _exact_oc(volfrac, rho, dcf)
    return phys, dc, comp, dcf, new, chg, vol, lam, steps


def _exact_run(pr, device):
    n, d = (pr.nelx, pr.nely), 2
    Ke = torch.from_numpy(compute_Ke_2d(pr.E, pr.nu)).to(device)
    shape = tuple(k + 1 for k in n) + (d,)
    f = torch.from_numpy(force_vector(pr)).to(device).reshape(shape)
    fixed = _fixed_bits(torch.from_numpy(fixed_node_mask(pr)).to(device), shape)
    rho = torch.full(n, float(pr.volfrac), dtype=torch.float64, device=device)
    u = torch.zeros_like(f)
    comp, vols = [], []
    for _ in range(pr.max_iter):
        phys = rho
        if pr.filter_type == "density":
            num, den = _exact_filter(n, pr.rmin, rho)
            phys = num / (den + 1e-20)
        scale = E_MIN + phys ** PENALTY * (1.0 - E_MIN)
        u = torch.where(fixed, torch.zeros_like(u), u)
        u, _ = _exact_pcg(n, Ke, None, 0.0, scale, f, fixed, u, pr.preconditioner,
                          pr.max_cg_iter, pr.cg_tol)
        _, _, co, _, rho, _, vol, _, _ = _exact_design(n, Ke, pr.rmin, pr.filter_type, rho, u,
                                                       pr.volfrac)
        comp.append(float(co))
        vols.append(vol)
    return rho, np.array(comp), np.array(vols)


def exact(case, seed):
    c = case
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    kind = c["kind"]
    if kind == "run":
        rho, comp, vol = _exact_run(_run_problem(c, np.random.default_rng(seed)), dev)
        return {"density": rho, "compliance": comp, "volume": vol}
    if kind == "batch":
        got = [_exact_run(p, dev) for p in _batch_problems(c, np.random.default_rng(seed))]
        return {"density": torch.cat([g[0].reshape(-1) for g in got]),
                "compliance": np.concatenate([g[1] for g in got])}
    n = (c["nx"], c["ny"]) + ((c["nz"],) if c["nz"] else ())
    d = len(n)
    Ke_np = compute_Ke_3d(1.0, 0.3) if d == 3 else compute_Ke_2d(1.0, 0.3)
    Ke = torch.from_numpy(Ke_np).to(dev)
    shape = tuple(k + 1 for k in n) + (d,)
    if kind == "solve":
        s = _solve_inputs(c, seed, dev)
        inv, alpha = regularized_inverse(Ke_np)
        scale = E_MIN + s["rho"].reshape(n) ** PENALTY * (1.0 - E_MIN)
        f = s["f"].reshape(shape)
        u, it = _exact_pcg(n, Ke, torch.from_numpy(np.asarray(inv)).to(dev), alpha, scale, f,
                           _fixed_bits(s["fixed"], shape), torch.zeros_like(f), c["pre"],
                           c["cg"], 1e-8)
        return {"u": u.reshape(-1), "iters": None}
    if kind == "design":
        s = _design_inputs(c, seed, dev)
        rho = s["rho"].reshape(n)
        phys, dc, comp, dcf, new, chg, vol, lam, steps = _exact_design(
            n, Ke, c["rmin"], c["filter"], rho, s["u"].reshape(shape), float(s["rho"].mean()))
        out = {"dc": dc.reshape(-1), "dcf": dcf.reshape(-1), "new": new.reshape(-1),
               "scalars": torch.tensor([float(comp), chg, vol, lam, float(steps)],
                                       dtype=torch.float64)}
        if c["filter"] == "density":
            out["phys"] = phys.reshape(-1)
        return out
    s = _matvec_inputs(c, seed, dev)
    p = s["p"].double().reshape(shape)
    scale = E_MIN + s["rho"].double().reshape(n) ** PENALTY * (1.0 - E_MIN)
    ap = torch.where(_fixed_bits(s["fixed"], shape), p, _apply(Ke, scale, p, n))
    return {"ap": ap.reshape(-1), "pap": (p * ap).sum().reshape(1)}
