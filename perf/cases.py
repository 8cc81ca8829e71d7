"""What is measured: the work a program has this library do, through its public entry points.

Kinds of case (every size is cells per axis, x fastest; fields are (nz, ny, nx)):

  solve   one homogenization from zero: update(k), heatMatrix(), Sensitivity(dC). 16^3 cells, where
          launches and latency count, to 256^3; cubes, flat and ragged boxes; FP32 and the two mixed
          forms; V(2,2) at 1e-6 and the library's default V(1,1) cycle.
  steps   a few iterations of an OC design loop from a new density: density chain and operators
          (update_density), the solve with K^H and the sensitivity, the filter adjoint and the OC
          update; the first solve starts from zero, the later ones from the previous solution.
  filter  the density chain and its adjoint on their own: odd sizes, both weights, both boundaries.
  oc      the sensitivity filter and the OC update on their own.
  mma     three steps of the method of moving asymptotes from a new point (the third is the first with
          moved asymptotes), one or two constraints.
  serve   a burst of independent requests of mixed sizes from host memory through the server.
  design  a short tensor-matching design run (run_custom) as the reference's main program makes it.
"""
import math

import numpy as np
import torch

from opentm_b200 import (DensityFilter, HomoConfig, Homogenization_H, MMAOptimizer, OCOptimizer, Server,
                         WEIGHT_LINEAR, WEIGHT_SPLINE4)
from opentm_b200.driver import DesignConfig, InitWay, Model, run_custom

P_SIMP, K0, KMIN = 3.0, 1.0, 1e-3
MIN_RHO, OC_STEP, OC_DAMP, VOLUME = 0.001, 0.02, 0.5, 0.3
DC = ((1.0, 0.3, -0.2), (0.1, -0.5, 0.25), (0.4, -0.15, 0.8))  # a tensor objective's derivative
TRACE = ((-1.0, 0.0, 0.0), (0.0, -1.0, 0.0), (0.0, 0.0, -1.0))  # the OC loop's objective -tr K^H
SERVE_SIZES = (32, 48, 64, 96)


def listed():
    return [
        # one small cell: a call is a chain of short launches
        {"name": "solve_32", "kind": "solve", "nx": 32, "ny": 32, "nz": 32, "field": "uniform", "precision": "fp32",
         "smooth": 2, "tol": 1e-6},
        # a cell whose axes are no multiples of a power of two above 8
        {"name": "solve_40x56x72", "kind": "solve", "nx": 40, "ny": 56, "nz": 72, "field": "uniform",
         "precision": "fp32", "smooth": 2, "tol": 1e-6},
        # the library's default cycle, V(1,1), on a flat box of a design-like field
        {"name": "solve_v11_96x128x64", "kind": "solve", "nx": 96, "ny": 128, "nz": 64, "field": "design",
         "precision": "fp32", "smooth": 1, "tol": 1e-6},
        # the mixed form: 16-bit fine level, FP64 solution, on a two-phase field
        {"name": "solve_128_bf16", "kind": "solve", "nx": 128, "ny": 128, "nz": 128, "field": "threshold",
         "precision": "bf16", "smooth": 2, "tol": 1e-6},
        # the largest solve: the working set is far above L2
        {"name": "solve_256", "kind": "solve", "nx": 256, "ny": 256, "nz": 256, "field": "threshold",
         "precision": "fp32", "smooth": 2, "tol": 1e-6},
        # the design loop most programs run: 128^3, warm-started after the first step
        {"name": "steps_128", "kind": "steps", "nx": 128, "ny": 128, "nz": 128, "steps": 3, "tol": 1e-6},
        # runCustom's filter (Spline4, radius 1.5, zero padding) on odd sizes
        {"name": "filter_100x75x131", "kind": "filter", "nx": 100, "ny": 75, "nz": 131, "weight": "spline4",
         "radius": 1.5, "periodic": False},
        # a wide periodic filter on a large cell
        {"name": "filter_256_r3", "kind": "filter", "nx": 256, "ny": 256, "nz": 256, "weight": "linear",
         "radius": 3.0, "periodic": True},
        # an OC iteration's sensitivity filter and update
        {"name": "oc_128", "kind": "oc", "nx": 128, "ny": 128, "nz": 128, "radius": 2.0},
        # MMA on a 128^3 cell's densities with one constraint, as the design driver uses it
        {"name": "mma_128", "kind": "mma", "n": 128 ** 3, "m": 1},
        # requests of mixed sizes from host memory, all at once
        {"name": "serve_24", "kind": "serve", "count": 24, "largest": 96},
        # a design run of ten OC iterations, solver set-up included
        {"name": "design_64", "kind": "design", "n": 64, "model": "oc", "iters": 10},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cell(rng, lo, hi):
    """Axes the multigrid hierarchy takes well (halved while all are even and at least 8): a base of
    4..13 per axis, at most 7^3 vertices together, times a power of two."""
    n = _log_int(rng, lo, hi)
    f = 1
    while n / (2 * f) > 7 and f < 32:
        f *= 2
    while True:
        base = [rng.randint(4, 13) if rng.random() < 0.6 else max(4, min(13, round(n / f))) for _ in range(3)]
        if base[0] * base[1] * base[2] <= 343 and max(base) * f <= hi:
            return [b * f for b in base]


def draw(rng):
    kind = rng.choices(("solve", "steps", "filter", "oc", "mma", "serve", "design"), (8, 4, 4, 2, 2, 1, 1))[0]
    if kind == "solve":
        nx, ny, nz = _cell(rng, 16, 192)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "field": rng.choice(("uniform", "threshold", "design")),
                "precision": rng.choice(("fp32", "fp32", "fp32", "bf16", "fp16")), "smooth": rng.choice((2, 2, 2, 1, 3)),
                "tol": 1e-6}
    if kind == "steps":
        nx, ny, nz = _cell(rng, 24, 144)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "steps": rng.randint(2, 3), "tol": 1e-6}
    if kind == "filter":
        radius = rng.choice((1.5, 2.0, 2.5, 3.0, 4.0))
        return {"kind": kind, "nx": _log_int(rng, 16, 256), "ny": _log_int(rng, 16, 256), "nz": _log_int(rng, 16, 256),
                "weight": rng.choice(("linear", "spline4")), "radius": radius, "periodic": rng.random() < 0.5}
    if kind == "oc":
        return {"kind": kind, "nx": _log_int(rng, 16, 192), "ny": _log_int(rng, 16, 192), "nz": _log_int(rng, 16, 192),
                "radius": rng.choice((1.5, 2.0, 2.0, 3.0))}
    if kind == "mma":
        return {"kind": kind, "n": _log_int(rng, 4096, 3000000), "m": rng.choice((1, 1, 2))}
    if kind == "serve":
        return {"kind": kind, "count": rng.randint(4, 32), "largest": rng.choice((48, 64, 96))}
    return {"kind": kind, "n": rng.choice((32, 48, 64, 80)), "model": rng.choice(("oc", "oc", "mma")),
            "iters": rng.randint(4, 10)}


# ---- inputs --------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _box_mean(a):
    for axis in range(3):
        a = (a + torch.roll(a, 1, axis) + torch.roll(a, -1, axis)) / 3.0
    return a


def _density(shape, field, gen):
    """uniform: i.i.d. densities; threshold: a smoothed normal field cut at its 40 % quantile (two
    phases with a sharp interface); design: a nearly even start of a design loop."""
    if field == "uniform":
        return 0.001 + 0.999 * torch.rand(shape, generator=gen, device="cuda")
    if field == "design":
        return 0.3 + 0.05 * (2.0 * torch.rand(shape, generator=gen, device="cuda") - 1.0)
    s = _box_mean(torch.randn(shape, generator=gen, device="cuda"))
    q = torch.sort(s.flatten()).values[int(0.4 * s.numel())]
    return torch.where(s >= q, s, torch.zeros_like(s)).clamp(0.001, 1.0)


def _simp(rho):
    return KMIN + rho ** 3 * (K0 - KMIN)


def _shape(case):
    return (case["nz"], case["ny"], case["nx"])


def _solve_inputs(case, seed):
    return _simp(_density(_shape(case), case["field"], _gen(seed))).contiguous()


def _filter_inputs(case, seed):
    g = _gen(seed)
    rho = 0.001 + 0.999 * torch.rand(_shape(case), generator=g, device="cuda")
    return rho, torch.randn(_shape(case), generator=g, device="cuda")


def _oc_inputs(case, seed):
    """A density in mid-loop and the (negative) sensitivities of -tr K^H, spread over two decades."""
    g = _gen(seed)
    rho = (0.3 + 0.2 * _box_mean(torch.randn(_shape(case), generator=g, device="cuda"))).clamp(MIN_RHO, 1.0)
    e = torch.exp(1.2 * torch.randn(_shape(case), generator=g, device="cuda"))
    return rho, -(e * rho ** 2 / rho.numel()).contiguous()


def _mma_inputs(case, seed):
    """The volume as objective and one or two weighted means to keep below a bound (the form in which
    the design driver poses a tensor match), with uneven weights."""
    n, m = case["n"], case["m"]
    g = _gen(seed)
    x = (0.1 + 0.5 * torch.rand(n, generator=g, device="cuda")).contiguous()
    dfdx = torch.full((n,), 1.0 / n, device="cuda")
    rows = [(-(0.2 + torch.rand(n, generator=g, device="cuda")) / n).contiguous() for _ in range(m)]
    return x, dfdx, rows, [0.05 + 0.02 * i for i in range(m)]


def _serve_inputs(case, seed):
    r = np.random.RandomState(seed % (1 << 31))
    sizes = [s for s in SERVE_SIZES if s <= case["largest"]]
    picked = [case["largest"]] + [int(s) for s in r.choice(sizes, case["count"] - 1)]
    g = _gen(seed)
    return [_simp(_box_mean(0.001 + 0.999 * torch.rand((n, n, n), generator=g, device="cuda"))).cpu().numpy()
            for n in picked]


def _design_density(case, seed):
    g = _gen(seed)
    return (0.5 + 0.3 * _box_mean(torch.randn((case["n"],) * 3, generator=g, device="cuda"))).clamp(0.1, 1.0)


# ---- the state a program keeps, and one pass -----------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("solve", "steps"):
        reso = (case["nx"], case["ny"], case["nz"])
        s["H"] = Homogenization_H(HomoConfig(reso=reso, femRelThres=case["tol"], pre_smooth=case.get("smooth", 2),
                                             post_smooth=case.get("smooth", 2), precision=case.get("precision", "fp32"),
                                             warm_start=kind == "steps"))
    if kind == "solve":
        s["k"] = _solve_inputs(case, seed)
        s["sens"] = torch.empty_like(s["k"])
        s["dC"] = np.array(DC)
    elif kind == "steps":
        s["rho0"] = _density(_shape(case), "design", _gen(seed)).contiguous()
        s["rho"], s["sens"], s["g"] = (torch.empty_like(s["rho0"]) for _ in range(3))
        s["df"] = DensityFilter(reso, 2.0, WEIGHT_LINEAR, True, P_SIMP, K0, KMIN)
        s["oc"] = OCOptimizer(s["rho"].numel(), MIN_RHO, OC_STEP, OC_DAMP)
        s["dC"] = np.array(TRACE)
    elif kind == "filter":
        weight = WEIGHT_SPLINE4 if case["weight"] == "spline4" else WEIGHT_LINEAR
        s["df"] = DensityFilter((case["nx"], case["ny"], case["nz"]), case["radius"], weight, case["periodic"], P_SIMP,
                                K0, KMIN)
        s["rho"], s["gk"] = _filter_inputs(case, seed)
        s["g"] = torch.empty_like(s["rho"])
    elif kind == "oc":
        s["rho0"], s["sens0"] = _oc_inputs(case, seed)
        s["rho"], s["sens"] = torch.empty_like(s["rho0"]), torch.empty_like(s["sens0"])
        s["oc"] = OCOptimizer(s["rho"].numel(), MIN_RHO, OC_STEP, OC_DAMP)
    elif kind == "mma":
        s["x0"], s["dfdx"], s["rows"], s["g"] = _mma_inputs(case, seed)
        s["x"] = torch.empty_like(s["x0"])
        s["mma"] = MMAOptimizer(case["m"], case["n"], 1.0, 0.0, 1000.0, 1.0)
        s["mma"].setBound(1e-4, 1.0)
    elif kind == "serve":
        s["k"] = _serve_inputs(case, seed)
        s["server"] = Server(hbm_budget_bytes=20 * 10 ** 9, fem_rel_thres=1e-6, pre_smooth=2, streams=8,
                             host_stage_bytes=1 << 28)
    else:
        s["rho0"] = _design_density(case, seed).cpu().numpy()
        s["config"] = DesignConfig(reso=case["n"], winit=InitWay.IWP, model=Model[case["model"]], max_iter=case["iters"],
                                   finthres=0.0)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "solve":
        s["H"].update(s["k"])
        C = s["H"].heatMatrix()
        s["H"].Sensitivity(s["dC"], s["sens"])
        return {"C": C, "sens": s["sens"]}
    if kind == "steps":
        s["rho"].copy_(s["rho0"])
        s["H"].reset_displacement()
        C = []
        for _ in range(case["steps"]):
            s["H"].update_density(s["df"], s["rho"])
            C.append(s["H"].heatMatrixSensitivity(s["dC"], s["sens"]))
            s["df"].backward(s["sens"], s["g"])
            s["oc"].update(s["g"], s["rho"], VOLUME)
        return {"C": C, "g": s["g"], "rho": s["rho"]}
    if kind == "filter":
        k = s["df"].forward(s["rho"])
        g = s["df"].backward(s["gk"], s["g"])
        return {"rho_f": s["df"].rho_f, "k": k, "dk": s["df"].dk, "g": g}
    if kind == "oc":
        s["rho"].copy_(s["rho0"])
        s["sens"].copy_(s["sens0"])
        s["oc"].filterSens(s["sens"], s["rho"], case["nx"], (case["nx"], case["ny"], case["nz"]), case["radius"])
        s["oc"].update(s["sens"], s["rho"], VOLUME)
        return {"sens": s["sens"], "rho": s["rho"]}
    if kind == "mma":
        s["x"].copy_(s["x0"])
        for itn in (1, 2, 3):
            s["mma"].update(itn, s["x"], s["dfdx"], s["g"], s["rows"])
        return {"x": s["x"]}
    if kind == "serve":
        ids = [s["server"].submit(k) for k in s["k"]]
        s["server"].run_until_idle()
        return {"C": [s["server"].poll(i)[0] for i in ids]}
    rho, info = run_custom(s["config"], s["rho0"])
    return {"rho": rho, "K": info["K"], "history": info["history"]}


# ---- what a pass cannot do without ---------------------------------------------------------------
def work(case):
    """Bytes: every input read once, every output written once. Operations: for a solve, the
    multigrid cycles that the tolerance takes (6 of them, each 2 * smooth sweeps and 3 operator
    products of 20 neighbours in 3 load cases on 8/7 of the vertices)."""
    kind = case["kind"]

    def solve_flops(nv, smooth, cycles):
        return cycles * (2 * smooth + 3) * 120.0 * nv * 8 / 7

    if kind in ("solve", "steps"):
        nv = case["nx"] * case["ny"] * case["nz"]
        steps = case.get("steps", 1)
        if kind == "solve":
            return {"bytes": 8.0 * nv, "flops": solve_flops(nv, case["smooth"], 6)}
        return {"bytes": 12.0 * nv * steps, "flops": solve_flops(nv, 2, 6 + 3 * (steps - 1))}
    if kind == "filter":
        nv = case["nx"] * case["ny"] * case["nz"]
        taps = 4.0 / 3.0 * math.pi * case["radius"] ** 3
        return {"bytes": 28.0 * nv, "flops": 4.0 * taps * nv}
    if kind == "oc":
        nv = case["nx"] * case["ny"] * case["nz"]
        taps = 4.0 / 3.0 * math.pi * case["radius"] ** 3
        return {"bytes": 16.0 * nv, "flops": (3.0 * taps + 20 * 6) * nv}
    if kind == "mma":  # x in and out, the gradients in; about 30 Newton steps of some 80 operations
        return {"bytes": 3 * 4.0 * (3 + case["m"]) * case["n"], "flops": 3 * 30 * (60.0 + 20 * case["m"]) * case["n"]}
    if kind == "serve":
        sizes = [n for n in SERVE_SIZES if n <= case["largest"]]
        nv = case["count"] * sum(n ** 3 for n in sizes) / len(sizes)
        return {"bytes": 4.0 * nv, "flops": solve_flops(nv, 2, 6)}
    nv = case["n"] ** 3
    return {"bytes": 12.0 * nv * case["iters"], "flops": case["iters"] * solve_flops(nv, 1, 2)}


def tolerance(case):
    kind = case["kind"]
    if kind == "solve":
        # the solver stops at a relative residual of 1e-6, which leaves an error that grows with the
        # square of the cell's size and is largest at single elements of a sharp interface
        return {"rel": 1e-5, "max": 2e-3}
    if kind == "steps":
        # as solve, and the OC bisection accepts any multiplier whose volume is within 1e-4
        return {"rel": 4e-4, "max": 2e-2}
    if kind == "filter":
        # 32-bit weights and sums of up to a few hundred taps: 1.8e-6 off the 64-bit values at radius 4
        return {"rel": 6e-6, "max": 1e-4}
    if kind == "oc":
        # 32-bit sums; a volume at the edge of the bisection's band of 1e-4 may stop it one step apart
        return {"rel": 1e-5, "max": 1e-3}
    if kind == "mma":
        return {"rel": 1e-6, "max": 1e-5}
    if kind == "serve":
        return {"rel": 5e-7, "max": 1e-6}
    # ten steps whose solves stop at a relative residual of 0.01 and whose densities move by at most
    # 0.02 a step
    return {"rel": 1e-2, "max": 0.3}


# ---- 64-bit results in plain torch ---------------------------------------------------------------
_CORNERS = [(b & 1, (b >> 1) & 1, b >> 2) for b in range(8)]
# element matrix of the trilinear cube Laplacian by the number of axes two nodes differ in
_BY_AXES = (1.0 / 3.0, 0.0, -1.0 / 12.0, -1.0 / 12.0)


def _element_matrix():
    ke = torch.tensor([[_BY_AXES[sum(p != q for p, q in zip(a, b))] for b in _CORNERS] for a in _CORNERS],
                      dtype=torch.float64, device="cuda")
    return ke


def _at_corner(u, c):
    """u at corner c of every element: element (x, y, z) holds the nodes (x..x+1, y..y+1, z..z+1)."""
    return torch.roll(u, (-c[2], -c[1], -c[0]), (-3, -2, -1))


def _macro():
    """The three unit macro fields at the 8 corners in the library's load-case order and signs:
    +y, -x, +z."""
    c = torch.tensor(_CORNERS, dtype=torch.float64, device="cuda")
    return torch.stack([c[:, 1], -c[:, 0], c[:, 2]], 0)  # (3 cases, 8 corners)


def _apply(k, ke, u):
    out = torch.zeros_like(u)
    corner = [_at_corner(u, c) for c in _CORNERS]
    total = sum(corner)
    for a, ca in enumerate(_CORNERS):
        # row a: 1/3 u_a - 1/12 (all corners but a and its three neighbours along one axis)
        near = [b for b, cb in enumerate(_CORNERS) if sum(p != q for p, q in zip(ca, cb)) == 1]
        v = corner[a] * (5.0 / 12.0) - (total - corner[near[0]] - corner[near[1]] - corner[near[2]]) / 12.0
        out += torch.roll(k * v, (ca[2], ca[1], ca[0]), (-3, -2, -1))
    return out


def _solve64(k32, x=None, tol=1e-10, most=6000):
    """The periodic fluctuations of the three load cases by Jacobi-preconditioned conjugate gradients."""
    k = k32.double() + 1e-9
    ke = _element_matrix()
    load = _macro() @ ke  # (3, 8)
    b = torch.zeros((3,) + tuple(k.shape), dtype=torch.float64, device="cuda")
    diag = torch.zeros_like(k)
    for a, c in enumerate(_CORNERS):
        back = (c[2], c[1], c[0])
        diag += torch.roll(k, back, (-3, -2, -1)) / 3.0
        for i in range(3):
            b[i] += torch.roll(k * load[i, a], back, (-3, -2, -1))
    b -= b.mean((1, 2, 3), keepdim=True)
    dot = lambda p, q: (p * q).sum((1, 2, 3), keepdim=True)  # noqa: E731
    x = torch.zeros_like(b) if x is None else x
    r = b - _apply(k, ke, x)
    z = r / diag
    z -= z.mean((1, 2, 3), keepdim=True)
    p, rz, bb = z.clone(), dot(r, z), dot(b, b)
    for it in range(most):
        q = _apply(k, ke, p)
        alpha = rz / dot(p, q).clamp_min(1e-300)
        x += alpha * p
        r -= alpha * q
        if it % 25 == 24 and bool((dot(r, r) <= tol * tol * bb).all()):
            break
        z = r / diag
        z -= z.mean((1, 2, 3), keepdim=True)
        new = dot(r, z)
        p = z + (new / rz.clamp_min(1e-300)) * p
        rz = new
    return x


def _energies(x):
    """(chi0 - chi)^T KE (chi0 - chi) per element for the pairs 00 01 02 11 12 22, over the volume in units
    where the cell is 1 wide in x (elements are cubes of side 1 / nx)."""
    macro, ke, ne = _macro(), _element_matrix(), x.shape[-1] ** 3
    w = [[float(macro[i, a]) - _at_corner(x[i], c) for a, c in enumerate(_CORNERS)] for i in range(3)]
    kw = [[sum(float(ke[a, b]) * w[i][b] for b in range(8) if float(ke[a, b])) for a in range(8)] for i in range(3)]
    return {(i, j): sum(w[i][a] * kw[j][a] for a in range(8)) / ne for i in range(3) for j in range(i, 3)}


def _tensor(k32, e):
    k = k32.double() + 1e-9
    C = np.zeros((3, 3))
    for (i, j), v in e.items():
        C[i, j] = C[j, i] = float((k * v).sum())
    return C


def _sens64(e, dC):
    return sum(v * (dC[i][j] + (dC[j][i] if i != j else 0.0)) for (i, j), v in e.items())


def _taps(weight, radius):
    h = int(radius + 0.5)
    out = {}
    for oz in range(-h, h + 1):
        for oy in range(-h, h + 1):
            for ox in range(-h, h + 1):
                q2 = (ox * ox + oy * oy + oz * oz) / radius ** 2
                q = math.sqrt(q2)
                w = 1 - 6 * q2 + 8 * q2 * q - 3 * q2 * q2 if weight == "spline4" else 1 - q
                if q2 < 1 and w:
                    out[(oz, oy, ox)] = w
    total = sum(out.values())
    return {o: w / total for o, w in out.items()}


def _moved(a, o, periodic):
    """b(i) = a(i + o), zero outside without periodicity."""
    if periodic:
        return torch.roll(a, (-o[0], -o[1], -o[2]), (0, 1, 2))
    out = torch.zeros_like(a)
    src, dst = [], []
    for n, d in zip(a.shape, o):
        lo, hi = max(0, -d), min(n, n - d)
        if hi <= lo:
            return out
        dst.append(slice(lo, hi))
        src.append(slice(lo + d, hi + d))
    out[tuple(dst)] = a[tuple(src)]
    return out


def _filter64(a, weight, radius, periodic):
    one = torch.ones_like(a)
    s, ws = torch.zeros_like(a), torch.zeros_like(a)
    for o, w in _taps(weight, radius).items():
        s += w * _moved(a, o, periodic)
        ws += w * _moved(one, o, periodic)
    return s / ws, ws


def _filter_adjoint64(g, ws, weight, radius, periodic):
    q, s = g / ws, torch.zeros_like(g)
    for o, w in _taps(weight, radius).items():
        s += w * _moved(q, tuple(-d for d in o), periodic)
    return s


def _oc64(sens, rho):
    """The OC update: bisection on the multiplier until the volume is within 1e-4 of its bound."""
    lo, hi = 0.0, float(sens.abs().max())
    new = rho
    for _ in range(20):
        g = float(np.float32((np.float32(lo) + np.float32(hi)) / np.float32(2)))
        B = -sens / g
        B = torch.where(B < 0, torch.full_like(B, 0.01), B)
        new = (rho * B ** OC_DAMP).clamp(rho - OC_STEP, rho + OC_STEP).clamp(MIN_RHO, 1.0)
        v = float(new.mean())
        if v < VOLUME - 1e-4:
            hi = g
        elif v > VOLUME + 1e-4:
            lo = g
        else:
            break
    return new


def _chain64(rho, weight, radius, periodic):
    f, ws = _filter64(rho, weight, radius, periodic)
    return f, ws, KMIN + (K0 - KMIN) * f ** 3, (K0 - KMIN) * 3 * f ** 2


def exact(case, seed):
    """The results in 64 bits, or None: a design run's own results (its solves stop at a relative
    residual of 0.01), the interior-point iterates of MMA and the largest solves have none here."""
    kind = case["kind"]
    if kind in ("solve", "steps") and case["nx"] * case["ny"] * case["nz"] > 2300000:
        return None
    if kind == "solve":
        k = _solve_inputs(case, seed)
        e = _energies(_solve64(k))
        return {"C": _tensor(k, e), "sens": _sens64(e, DC)}
    if kind == "steps":
        rho = _density(_shape(case), "design", _gen(seed)).double()
        C, x, g = [], None, None
        for _ in range(case["steps"]):
            _, ws, k, dk = _chain64(rho, "linear", 2.0, True)
            x = _solve64(k, x)
            e = _energies(x)
            C.append(_tensor(k, e))
            g = _filter_adjoint64(_sens64(e, TRACE) * dk, ws, "linear", 2.0, True)
            rho = _oc64(g, rho)
        return {"C": C, "g": g, "rho": rho}
    if kind == "filter":
        rho, gk = _filter_inputs(case, seed)
        how = (case["weight"], case["radius"], case["periodic"])
        f, ws, k, dk = _chain64(rho.double(), *how)
        return {"rho_f": f, "k": k, "dk": dk, "g": _filter_adjoint64(gk.double() * dk, ws, *how)}
    if kind == "oc":
        rho, sens = (t.double() for t in _oc_inputs(case, seed))
        s, w = torch.zeros_like(rho), 0.0
        for o, c in _taps("linear", case["radius"]).items():
            s += c * _moved(sens * rho, o, True)
            w += c
        s = s / (w * rho)
        return {"sens": s, "rho": _oc64(s, rho)}
    if kind == "serve":
        out = []
        for k in _serve_inputs(case, seed):
            kd = torch.from_numpy(k).cuda()
            out.append(_tensor(kd, _energies(_solve64(kd))))
        return {"C": out}
    return None
