"""The performance cases of the framework: what a simulation has it do.

Each case is one call, or one short sequence of calls, of the public entry
points on the data such a program holds on the GPU at that moment.  The
sizes are those of the benchmark workloads (bench.py) and of the tests, and
ranges around them:

* ``pairs``: the all-pairs sums of ``fiber3d_b200.kernels``, the hot path of
  every matvec;
* ``fiber_inverse`` / ``fiber_lu``: the fiber blocks of the GMRES
  preconditioner, rebuilt as the fibers move (``blocklu.BlockLU``);
* ``quadrature``: the RBF surface quadrature of a periphery (set-up);
* ``shell_inverse``: the dense periphery or body preconditioner (set-up);
* ``fmm``: the fast multipole sums of runs with useFMM, the points new at
  every time step and the sums evaluated once per GMRES matvec;
* ``step``: one implicit time step, right-hand side, preconditioner and solve.

``listed`` and ``draw`` give the cases, ``prepare`` makes a case's inputs from
a seed, ``run`` is one pass, ``work`` what the pass cannot do without, and
``exact`` the same outputs in 64-bit torch without this package.
"""
import math

import numpy as np
import torch

from fiber3d_b200 import fmm, geometry, hydro, kernels
from fiber3d_b200.blocklu import BlockLU
from fiber3d_b200.quadrature import surface_quadrature_weights

ETA, REG, EPS = 1.0, 5e-3, 1e-5  # the drop-ins' defaults
RADIUS = 10.0                    # of the periphery
FIBER_SIZES = (16, 24, 32, 48, 64)


def listed():
    return [
        # the smallest sum the benchmark has: 32 fibers of 32 points, latency and launches count
        {"name": "oseen_1024", "kind": "pairs", "kernel": "oseen", "sources": 1024, "targets": 0, "precision": "fp64"},
        # the periphery's double layer on itself and on points of the volume, as GMRES and post-processing evaluate it
        {"name": "stresslet_12000", "kind": "pairs", "kernel": "stresslet", "sources": 12000, "targets": 4096,
         "precision": "fp64"},
        # the same in the inner solves' precision
        {"name": "stresslet_12000_fp32c", "kind": "pairs", "kernel": "stresslet", "sources": 12000, "targets": 4096,
         "precision": "fp32c"},
        # 512 fibers of 32 points: the blocks' inverses and one application, each time step
        {"name": "fiber_inverse_512x32", "kind": "fiber_inverse", "fibers": 512, "points": 32, "precision": "fp64"},
        # 2000 fibers of mixed resolution: factorisation and one substitution
        {"name": "fiber_lu_2000", "kind": "fiber_lu", "fibers": 2000, "points": 0},
        # a coarse and a full periphery
        {"name": "quadrature_1442", "kind": "quadrature", "frequency": 12},
        {"name": "quadrature_12252", "kind": "quadrature", "frequency": 35},
        # a rigid body's surface and a mid-sized periphery
        {"name": "shell_inverse_400", "kind": "shell_inverse", "nodes": 400},
        {"name": "shell_inverse_3000", "kind": "shell_inverse", "nodes": 3000},
        # single and double layer at as many targets, the benchmark's smaller and larger sizes
        {"name": "fmm_1e5", "kind": "fmm", "points": 100000, "order": 8, "evaluations": 2},
        {"name": "fmm_1e6", "kind": "fmm", "points": 1000000, "order": 8, "evaluations": 2},
        # 512 fibers, 4 bodies of 400 nodes, a periphery of 6000: the time step in double precision
        {"name": "step_512", "kind": "step", "fibers": 512, "bodies": 4, "nodes": 6000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pairs", "pairs", "pairs", "fiber_inverse", "fiber_lu", "quadrature", "shell_inverse", "fmm",
                       "fmm", "step"])
    if kind == "pairs":
        return {"kind": kind, "kernel": rng.choice(["oseen", "stresslet", "rotlet"]), "sources": _log(rng, 300, 24000),
                "targets": rng.choice([0, _log(rng, 100, 8000)]), "precision": rng.choice(["fp64", "fp64", "fp32c"])}
    if kind == "fiber_inverse":
        return {"kind": kind, "fibers": _log(rng, 20, 2000), "points": rng.choice([8, 16, 24, 32]),
                "precision": rng.choice(["fp64", "fp32c"])}
    if kind == "fiber_lu":
        return {"kind": kind, "fibers": _log(rng, 20, 2000), "points": rng.choice([0, 0, 32, 48, 64])}
    if kind == "quadrature":
        return {"kind": kind, "frequency": _log(rng, 8, 40)}
    if kind == "shell_inverse":
        return {"kind": kind, "nodes": _log(rng, 100, 3000)}
    if kind == "fmm":
        return {"kind": kind, "points": _log(rng, 30000, 800000), "order": rng.choice([6, 8]),
                "evaluations": rng.randint(1, 2)}
    return {"kind": kind, "fibers": _log(rng, 16, 512), "bodies": rng.randint(0, 4), "nodes": _log(rng, 400, 4000)}


# ------------------------------------------------------------------ inputs --
def _dev(a):
    return torch.as_tensor(a, device="cuda").contiguous()


def _fiber_counts(case):
    """Points of each fiber: the case's, or (0) a mix, the same whatever the seed."""
    n = case["fibers"]
    return np.random.default_rng(n).choice(FIBER_SIZES, size=n) if case["points"] == 0 else [case["points"]] * n


def _sphere_mesh(f, rng):
    """Nodes (10 f^2 + 2) and triangles (20 f^2) of an icosahedron whose
    edges are divided by f, on the sphere of radius RADIUS, the nodes moved
    along the surface by up to a tenth of their spacing."""
    p = (1.0 + math.sqrt(5.0)) / 2.0
    v = np.array([(-1, p, 0), (1, p, 0), (-1, -p, 0), (1, -p, 0), (0, -1, p), (0, 1, p), (0, -1, -p), (0, 1, -p),
                  (p, 0, -1), (p, 0, 1), (-p, 0, -1), (-p, 0, 1)]) / math.sqrt(1.0 + p * p)
    faces = [(0, 11, 5), (0, 5, 1), (0, 1, 7), (0, 7, 10), (0, 10, 11), (1, 5, 9), (5, 11, 4), (11, 10, 2),
             (10, 7, 6), (7, 1, 8), (3, 9, 4), (3, 4, 2), (3, 2, 6), (3, 6, 8), (3, 8, 9), (4, 9, 5), (2, 4, 11),
             (6, 2, 10), (8, 6, 7), (9, 8, 1)]
    ids, points, tri = {}, [], []

    def node(a, b, c, i, j):  # (f - i - j) a + i b + j c, the same node on a shared edge
        key = tuple(sorted((q, w) for q, w in ((a, f - i - j), (b, i), (c, j)) if w))
        if key not in ids:
            ids[key] = len(points)
            points.append(sum(w * v[q] for q, w in key))
        return ids[key]

    for a, b, c in faces:
        at = [[node(a, b, c, i, j) for j in range(f + 1 - i)] for i in range(f + 1)]
        for i in range(f):
            for j in range(f - i):
                tri.append((at[i][j], at[i + 1][j], at[i][j + 1]))
                if i + j < f - 1:
                    tri.append((at[i + 1][j], at[i + 1][j + 1], at[i][j + 1]))
    x = np.array(points)
    x /= np.linalg.norm(x, axis=1, keepdims=True)
    x += rng.uniform(-0.06, 0.06, size=x.shape) / f
    x *= RADIUS / np.linalg.norm(x, axis=1, keepdims=True)
    return x, np.array(tri, dtype=np.int32)


def _fiber_blocks(case, rng):
    """The fiber blocks of a time step at the fibers' positions, as the
    assembly of that step leaves them on the GPU."""
    counts = _fiber_counts(case)
    fibers = geometry.perturbed_fibers(rng, case["fibers"], counts, 2.0, RADIUS)
    forces = np.concatenate([np.tile(rng.normal(scale=0.1, size=3), (n, 1)) for n in counts])
    system = hydro.HydroSystem(hydro.Problem(fibers, [2.0] * case["fibers"], 0.0025, 1e-3, 1.0, [], None, forces))
    lu = BlockLU([4 * int(n) for n in counts])
    return {"lu": lu, "blocks": system.A_fib[:lu.A.numel()].clone(), "rhs": _dev(rng.normal(size=lu.nvec))}


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    state = {"case": case}
    if kind == "pairs":
        n = case["sources"]
        if case["kernel"] == "oseen":
            x = geometry.straight_fibers_cheb(rng, -(-n // 32), 32, 2.0, 5.0)[:n]
            normals = x
        else:
            x, normals = geometry.fibonacci_sphere(n + n % 2, RADIUS)
            x, normals = x[:n], normals[:n]
        state.update(x=_dev(x), normals=_dev(normals), density=_dev(rng.normal(size=(n, 3))),
                     targets=_dev(geometry.uniform_ball(rng, case["targets"], 0.9 * RADIUS)))
    elif kind in ("fiber_inverse", "fiber_lu"):
        state.update(_fiber_blocks(case, rng))
        state.update(y=torch.empty_like(state["rhs"]))
    elif kind == "quadrature":
        x, tri = _sphere_mesh(case["frequency"], rng)
        state.update(nodes=_dev(x), triangles=_dev(tri), gradient=_dev(2.0 * x))
    elif kind == "shell_inverse":
        x, normals, w = _shell(case, rng)
        state.update(op=hydro.ShellOperator(hydro.Shell(x, -normals, w), build_inverse=False))
    elif kind == "fmm":
        n = case["points"]
        side = (4.0 * math.pi * 2 * n / (3 * 1e-3)) ** (1.0 / 3.0)
        gen = torch.Generator(device="cuda").manual_seed(seed)
        new = lambda f: f((n, 3), dtype=torch.float64, device="cuda", generator=gen)
        state.update(handle=fmm.FMM(order=case["order"], max_pts=1000), sl=new(torch.rand) * side,
                     dl=new(torch.rand) * side, trg=new(torch.rand) * side, normal=new(torch.randn),
                     densities=[(new(torch.randn), new(torch.randn)) for _ in range(case["evaluations"])])
    else:
        problem = geometry.hydro_step_problem(seed=seed, nfib=case["fibers"], nbody=case["bodies"],
                                              nshell=case["nodes"] - case["nodes"] % 2)
        state.update(system=hydro.HydroSystem(problem, tune=True))
    return state


def _shell(case, rng):
    """A Fibonacci sphere of the case's nodes (even), its weights a little uneven."""
    n = case["nodes"] - case["nodes"] % 2
    x, normals = geometry.fibonacci_sphere(n, RADIUS)
    return x, normals, 4.0 * math.pi * RADIUS ** 2 / n * rng.uniform(0.95, 1.05, size=n)


# --------------------------------------------------------------- one pass --
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "pairs":
        x, t, d, n, p = state["x"], state["targets"], state["density"], state["normals"], case["precision"]
        out = []
        if case["kernel"] == "oseen":
            out.append(kernels.oseen_kernel_times_density_numba(x, d, precision=p))
            if case["targets"]:
                out.append(kernels.oseen_kernel_source_target_numba(x, t, d, precision=p))
        elif case["kernel"] == "stresslet":
            out.append(kernels.stresslet_kernel_times_normal_times_density_numba(x, n, d, precision=p))
            if case["targets"]:
                out.append(kernels.stresslet_kernel_source_target_numba(x, t, n, d, precision=p))
        else:
            out.append(kernels.rotlet_kernel_source_target_numba(x, t if case["targets"] else x, d, precision=p))
        return out
    if kind == "fiber_inverse":
        lu = state["lu"]
        lu.A.copy_(state["blocks"])
        lu.invert(fp32=case["precision"] != "fp64")
        lu.apply(state["rhs"], state["y"], case["precision"])
        return {"inverses": lu.A if case["precision"] == "fp64" else lu.A32, "solution": state["y"]}
    if kind == "fiber_lu":
        lu = state["lu"]
        lu.A.copy_(state["blocks"])
        lu.factor()
        state["y"].copy_(state["rhs"])
        lu.solve(state["y"])
        return {"factors": lu.A, "pivots": lu.piv, "solution": state["y"]}
    if kind == "quadrature":
        return surface_quadrature_weights(state["nodes"], state["triangles"], state["gradient"])
    if kind == "shell_inverse":
        state["op"].build_inverse()
        return state["op"].inv64
    if kind == "fmm":
        h = state["handle"]
        h.set_points(state["sl"], state["dl"], state["trg"])
        return [h.evaluate(sl_density=f, dl_normal=state["normal"], dl_density=d) for f, d in state["densities"]]
    system = state["system"]
    system.update()
    solved = system.solve(tol=1e-10)
    return {"rhs": system.rhs, "x": solved["x"], "blocks": system.A_fib, "inverses": system.lu.A}


# ----------------------------------------------------------- what it needs --
def work(case):
    kind = case["kind"]
    if kind == "pairs":
        ns, nt = case["sources"], case["targets"]
        if case["kernel"] == "rotlet":
            pairs, read, per, points = ns * (nt or ns), 48 * ns, 25, nt or ns
        else:
            pairs, points = ns * (ns - 1) + ns * nt, ns + nt
            read, per = (72, 29) if case["kernel"] == "stresslet" else (48, 28)
            read *= ns
        return {"bytes": read + 24 * nt + 24 * points, "flops": float(per) * pairs}
    if kind in ("fiber_inverse", "fiber_lu"):
        mean = lambda k: sum((4.0 * n) ** k for n in FIBER_SIZES) / len(FIBER_SIZES) \
            if case["points"] == 0 else (4.0 * case["points"]) ** k
        b, n1, n2, n3 = case["fibers"], mean(1), mean(2), mean(3)
        if kind == "fiber_lu":
            return {"bytes": b * (16 * n2 + 20 * n1), "flops": b * (2.0 / 3.0 * n3 + 2 * n2)}
        out = 8 if case["precision"] == "fp64" else 12
        return {"bytes": b * ((8 + out) * n2 + 16 * n1), "flops": b * (2.0 * n3 + 2 * n2)}
    if kind == "quadrature":
        f = case["frequency"]
        nodes, tri, m = 10 * f * f + 2, 20 * f * f, 116
        return {"bytes": 56.0 * nodes + 12.0 * tri, "flops": tri * (2.0 / 3.0 * m ** 3 + 2.0 * m * m)}
    if kind == "shell_inverse":
        m = 3.0 * (case["nodes"] - case["nodes"] % 2)
        return {"bytes": 14 * m * m + 56 * m, "flops": 2 * m ** 3}
    if kind == "fmm":
        n = float(case["points"])
        depth = 2
        while 2 * n > 1000 * 8 ** depth:
            depth += 1
        # the near field alone: 27 leaves of both layers per target
        near = n * 27 * n / 8 ** depth * (28 + 29)
        return {"bytes": n * (72 + case["evaluations"] * (72 + 24)), "flops": case["evaluations"] * near}
    n, b, s = 32.0 * case["fibers"], 400.0 * case["bodies"], float(case["nodes"])
    # the explicit flow, and four iterations of the matvec and the preconditioner
    pairs = n * (n + b + s) * 28 * 5 + (b + s) * (n + b + s) * 29 * 4
    blocks = case["fibers"] * 128.0 ** 2
    return {"bytes": 8 * (4 * 9 * s * s + 8 * blocks), "flops": pairs + case["fibers"] * 2 * 128.0 ** 3}


# ------------------------------------------------------- the same in torch --
def _pair_sum(kernel, xs, xt, dens, normal, skip_self):
    """All pairs of sources xs and targets xt; a pair closer than EPS takes
    sqrt(r^2 + REG^2) for its distance, with skip_self i == j is left out."""
    out = torch.empty_like(xt)
    step = max(1, 20_000_000 // max(1, xs.shape[0]))
    for a in range(0, xt.shape[0], step):
        r = [xt[a:a + step, c, None] - xs[None, :, c] for c in range(3)]
        r2 = r[0] * r[0] + r[1] * r[1] + r[2] * r[2]
        r2 = torch.where(r2 < EPS * EPS, r2 + REG * REG, r2)
        inv = r2.rsqrt()
        if skip_self:
            k = torch.arange(inv.shape[0], device=inv.device)
            inv[k, k + a] = 0.0
        rd = r[0] * dens[:, 0] + r[1] * dens[:, 1] + r[2] * dens[:, 2]
        for c in range(3):
            if kernel == "oseen":
                v = (inv * dens[:, c] + inv ** 3 * rd * r[c]).sum(1) / (8.0 * math.pi * ETA)
            elif kernel == "rotlet":
                p, q = (c + 1) % 3, (c + 2) % 3
                v = (inv ** 3 * (dens[:, p] * r[q] - dens[:, q] * r[p])).sum(1) / (8.0 * math.pi * ETA)
            else:
                rn = r[0] * normal[:, 0] + r[1] * normal[:, 1] + r[2] * normal[:, 2]
                v = (inv ** 5 * rd * rn * r[c]).sum(1) * (-3.0 / (4.0 * math.pi * ETA))
            out[a:a + step, c] = v
    return out.reshape(-1)


def _cross(a, b):
    return torch.linalg.cross(a, b, dim=-1)


def _dot(a, b):
    return (a * b).sum(-1)


def _unit(a):
    return a / a.norm(dim=-1, keepdim=True)


def _quadrature(nodes, triangles, gradient):
    """The RBF quadrature weights of a closed surface (Reeger, Fornberg and
    Watts, Proc. R. Soc. A 472, 2016: r^7 and degree-7 polynomials on the 80
    nearest nodes of each triangle), in blocks of triangles."""
    tri = triangles.long().sort(dim=1).values
    count = tri.shape[0]
    corner = nodes[tri]
    normal = _unit(_cross(corner[:, 1] - corner[:, 0], corner[:, 2] - corner[:, 0]))
    # normals of the edges (0,1), (0,2), (1,2): the mean of the two triangles'
    ends = torch.stack([tri[:, [0, 1]], tri[:, [0, 2]], tri[:, [1, 2]]], 1).reshape(-1, 2)
    order = torch.argsort(ends[:, 0] * nodes.shape[0] + ends[:, 1], stable=True)
    first, second = order[0::2], order[1::2]
    na, nb = normal[first // 3], normal[second // 3]
    mean = _unit(na + torch.sign(_dot(na, nb))[:, None] * nb)
    edge = torch.empty((3 * count, 3), dtype=nodes.dtype, device=nodes.device)
    edge[first], edge[second] = mean, mean
    edge = edge.view(count, 3, 3)
    gx, gw = (torch.as_tensor(a, device=nodes.device) for a in np.polynomial.legendre.leggauss(6))
    gt, gw = 0.5 * (gx + 1.0), 0.5 * gw
    weights = torch.zeros(nodes.shape[0], dtype=nodes.dtype, device=nodes.device)
    for s in range(0, count, 2048):
        A, B, C = corner[s:s + 2048].unbind(1)
        n, (e_ab, e_ca, e_bc) = normal[s:s + 2048], edge[s:s + 2048].unbind(1)
        mid = (A + B + C) / 3
        near = ((mid[:, None] - nodes[None]) ** 2).sum(-1).topk(80, largest=False).indices
        v_oa = _cross(_cross(e_ab, B - A), _cross(e_ca, A - C))
        o_bc = _cross(e_bc, C - B)
        origin = A + (_dot(o_bc, B - A) / _dot(o_bc, v_oa))[:, None] * v_oa  # the projection's centre
        # in the triangle's plane, about its midpoint
        rxy, z = n[:, :2].norm(dim=1), torch.zeros_like(n[:, 0])
        e1 = torch.stack([n[:, 2] * n[:, 0] / rxy, n[:, 2] * n[:, 1] / rxy, -rxy], 1)
        e2 = torch.stack([-n[:, 1] / rxy, n[:, 0] / rxy, z], 1)
        plane = lambda p: torch.stack([_dot(p, e1[:, None]), _dot(p, e2[:, None])], -1)
        q = nodes[near]
        ray = q - origin[:, None]
        p = q + (_dot(n[:, None], A[:, None] - q) / _dot(n[:, None], ray))[..., None] * ray - origin[:, None]
        shift = plane((mid - origin)[:, None])
        height = _dot(p[:, 0], n)
        c = plane(p) - shift
        v = plane(torch.stack([A, B, C], 1) - origin[:, None]) - shift
        sign = torch.sign((v[:, 1, 0] - v[:, 0, 0]) * (v[:, 2, 1] - v[:, 0, 1]) -
                          (v[:, 1, 1] - v[:, 0, 1]) * (v[:, 2, 0] - v[:, 0, 0]))
        # integrals over the triangle of r^7 about each node and of the monomials
        rbf, poly = torch.zeros_like(c[..., 0]), []
        for k in range(3):
            p1, p2 = v[:, k, None], v[:, (k + 1) % 3, None]
            e = p2 - p1
            foot = (_dot(c - p1, e) / _dot(e, e))[..., None] * e + p1
            a = (c - foot).norm(dim=-1)
            for from_, to in ((p1, foot), (foot, p2)):
                turn = torch.sign((to - c)[..., 1] * (from_ - c)[..., 0] - (to - c)[..., 0] * (from_ - c)[..., 1])
                b = (to - from_).norm(dim=-1)
                a2, b2 = a * a, b * b
                part = a * (b * (a2 + b2).sqrt() * (279 * a2 ** 3 + 326 * a2 * a2 * b2 + 200 * a2 * b2 * b2 +
                                                    48 * b2 ** 3) + 105 * a2 ** 4 * torch.asinh(b / a)) / 3456
                rbf += torch.where((a > 0) & (b > 0), sign[:, None] * turn * part, torch.zeros_like(part))
        powers = [(d - k, k) for d in range(8) for k in range(d + 1)]
        for i, j in powers:
            total = torch.zeros_like(sign)
            for k in range(3):
                p1, p2 = v[:, k], v[:, (k + 1) % 3]
                x = p1[:, :1] + gt * (p2 - p1)[:, :1]
                y = p1[:, 1:] + gt * (p2 - p1)[:, 1:]
                total += (p2 - p1)[:, 1] * (gw * x ** (i + 1) * y ** j).sum(1) / (i + 1)
            poly.append(sign * total)
        m = torch.zeros((len(A), 116, 116), dtype=nodes.dtype, device=nodes.device)
        ip = c @ c.transpose(1, 2)
        d = ip.diagonal(dim1=1, dim2=2)
        m[:, :80, :80] = ((d[:, :, None] + d[:, None] - 2 * ip) ** 7).sqrt()
        P = torch.stack([c[..., 0] ** i * c[..., 1] ** j for i, j in powers], -1)
        m[:, :80, 80:], m[:, 80:, :80] = P, P.transpose(1, 2)
        rhs = torch.cat([rbf, torch.stack(poly, 1)], 1)
        w = torch.linalg.solve(m, rhs[..., None])[:, :80, 0]
        # area of the surface for area of the plane
        far = ray.norm(dim=-1)
        flat = (((c + shift) ** 2).sum(-1) + height[:, None] ** 2).sqrt()
        to = ray / far[..., None]
        w = w * (_dot(to, n[:, None]) / _dot(_unit(gradient[near]), to) * (far / flat) ** 2).abs()
        weights.index_add_(0, near.reshape(-1), w.reshape(-1))
    return weights


def _shell_inverse(case, seed):
    """Inverse of the periphery's dense double-layer operator: off the
    diagonal the stresslet times the source normal, its unit-density sums (the
    singularity vectors) and the identity over the weight taken from the
    diagonal, the rank-one normal term added."""
    x, normals, w = (_dev(a) for a in _shell(case, np.random.default_rng(seed)))
    normals = -normals
    n = x.shape[0]
    m = torch.zeros((n, 3, n, 3), dtype=torch.float64, device="cuda")
    r = x[:, None] - x[None]
    r2 = (r * r).sum(-1)
    r2.fill_diagonal_(1.0)
    f = -3.0 / (4.0 * math.pi * ETA) * (r * normals[None]).sum(-1) * r2 ** -2.5
    f.fill_diagonal_(0.0)
    for a in range(3):
        for b in range(3):
            m[:, a, :, b] = f * r[..., a] * r[..., b]
    k = torch.arange(n, device="cuda")
    unit = torch.einsum("iajb,j->iab", m, w) + torch.eye(3, dtype=torch.float64, device="cuda")
    m[k, :, k, :] -= unit / w[:, None, None]
    m = m.view(3 * n, 3 * n)
    m += torch.outer(normals.reshape(-1), normals.reshape(-1))
    return torch.linalg.inv(m)


def exact(case, seed):
    kind = case["kind"]
    if kind == "step" or (kind == "fmm" and case["points"] > 200000):
        return None
    if kind == "shell_inverse":
        return _shell_inverse(case, seed)
    state = prepare(case, seed)
    if kind == "pairs":
        x, t, d, n = state["x"], state["targets"], state["density"], state["normals"]
        if case["kernel"] == "rotlet":
            return [_pair_sum("rotlet", x, t if case["targets"] else x, d, None, False)]
        out = [_pair_sum(case["kernel"], x, x, d, n, True)]
        return out + [_pair_sum(case["kernel"], x, t, d, n, False)] if case["targets"] else out
    if kind in ("fiber_inverse", "fiber_lu"):
        lu, x = state["lu"], torch.empty_like(state["rhs"])
        first = torch.empty_like(state["blocks"])
        for b in range(lu.count):
            n, o, v = int(lu.sizes_h[b]), int(lu.moff_h[b]), int(lu.voff_h[b])
            m = state["blocks"][o:o + n * n].view(n, n).cpu()
            rhs = state["rhs"][v:v + n, None].cpu()
            if kind == "fiber_inverse":
                result = torch.linalg.inv(m)
                x[v:v + n] = (result @ rhs)[:, 0]
            else:
                result, pivots = torch.linalg.lu_factor(m)
                x[v:v + n] = torch.linalg.lu_solve(result, pivots, rhs)[:, 0]
            first[o:o + n * n] = result.reshape(-1)
        if kind == "fiber_inverse":
            return {"inverses": first, "solution": x}
        return {"factors": first, "pivots": None, "solution": x}
    if kind == "quadrature":
        return _quadrature(state["nodes"], state["triangles"], state["gradient"])
    out = []
    for f, d in state["densities"]:
        out.append(_pair_sum("oseen", state["sl"], state["trg"], f, None, False) +
                   _pair_sum("stresslet", state["dl"], state["trg"], d, state["normal"], False))
    return out
