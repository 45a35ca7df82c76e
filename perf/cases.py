"""The framework's work as performance cases: what is timed when its kernels change.

A case is one call, or the few calls that a design-optimisation program makes one after the
other, through the public entry points, at sizes from the smallest test mesh to the benchmark
mesh.  `listed()` names the fixed cases, `draw(rng)` gives more of the same ranges,
`prepare(case, seed)` makes what a program holds before the call (mesh handle, fields,
parameters), `run(state)` is one pass, `work(case)` the bytes and operations a pass cannot do
without, and `exact(case, seed)` the pass's results in 64 bits by plain torch.

Meshes are boxes [0,2]x[0,1]x[0,1] of nx x ny x nz hexes cut into 6 tetrahedra each
(numbered x slowest, z fastest), clamped on x = 0 and loaded with a traction on x = 2; a
jittered mesh has its interior nodes moved by up to 0.15 of the spacing, so that no two cells
are alike.
"""
import math

import numpy as np
import torch

# the 6 tetrahedra of a hex around its (0,0,0)-(1,1,1) diagonal
RING = ((1, 1, 0), (0, 1, 0), (0, 1, 1), (0, 0, 1), (1, 0, 1), (1, 0, 0))
NU, PENALTY, RHO_MIN = 0.3, 3.0, 1e-9
LAMBDA, MU = NU / ((1 + NU) * (1 - 2 * NU)), 0.5 / (1 + NU)
BATCH_SIZES = (16, 24, 32, 48, 64)
# (input channels, output channels, taps) of the warm-start network's layers
LAYERS = ((16, 16, 27), (16, 16, 27), (16, 32, 27), (32, 32, 27), (32, 64, 27), (64, 64, 27),
          (96, 32, 27), (32, 32, 27), (48, 16, 27), (16, 16, 27), (16, 9, 1))


def listed():
    return [
        # the smallest call of an optimiser or a line search: the residual of the 12,000-tet
        # cantilever, where the launches count
        {"name": "residual_small", "op": "residual", "nx": 20, "ny": 10, "nz": 10, "jitter": False},
        # the residual on the benchmark mesh (6.1 M tets)
        {"name": "residual_large", "op": "residual", "nx": 160, "ny": 80, "nz": 80, "jitter": False},
        # the 3x3 block Jacobian that a caller hands to its own solver, 2.6 M tets
        {"name": "jacobian_large", "op": "jacobian", "nx": 120, "ny": 60, "nz": 60, "jitter": False},
        # the pieces of an explicit adjoint on a general mesh of odd size: df/du and
        # df/dz + (dR/dz)^T lambda
        {"name": "adjoint_ragged", "op": "adjoint", "nx": 61, "ny": 37, "nz": 29, "jitter": True},
        # compliance and dC/dz of a converged design step, the benchmark mesh
        {"name": "criterion_large", "op": "criterion", "nx": 160, "ny": 80, "nz": 80, "jitter": False},
        # the operator without a matrix, as the matrix-free Krylov method applies it
        {"name": "matrix_free_apply", "op": "matrix_free", "nx": 90, "ny": 44, "nz": 46, "jitter": False},
        # one optimisation step of the 12,000-tet cantilever with the plain Jacobi-PCG
        {"name": "step_small_plain", "op": "step", "method": "plain", "nx": 20, "ny": 10, "nz": 10, "host": False},
        # one step on host buffers (the MPMD sequence) at a middle size, FP32 two-level method
        {"name": "step_host_middle", "op": "step", "method": "two-level", "nx": 60, "ny": 30, "nz": 30, "host": True},
        # the headline: one step of the 3.2 M-dof cantilever, FP16 two-level method
        {"name": "step_large", "op": "step", "method": "two-level-fp16", "nx": 160, "ny": 80, "nz": 80, "host": False},
        # the density filter around every step: filtered density and the chain rule back
        {"name": "filter_middle", "op": "filter", "nx": 80, "ny": 40, "nz": 40, "length": 0.05},
        # many designs and load cases at once
        {"name": "batch", "op": "batch", "count": 12},
        # a training step of the warm-start network on its own grid, batch 8
        {"name": "network_train", "op": "train", "n0": 65, "n1": 33, "n2": 33, "batch": 8},
    ]


def _size(rng, low, high):
    """A box of about n x n/2 x n/2 hexes, n spread over its logarithm, odd numbers among them."""
    n = math.exp(rng.uniform(math.log(low), math.log(high)))
    return {"nx": max(2, round(n)), "ny": max(2, round(n / 2 * rng.uniform(0.85, 1.0))),
            "nz": max(2, round(n / 2 * rng.uniform(0.85, 1.0)))}


def draw(rng):
    op = rng.choice(("residual", "jacobian", "adjoint", "criterion", "matrix_free", "step", "step", "step",
                     "filter", "batch", "train", "forward"))
    if op in ("residual", "adjoint", "criterion", "matrix_free"):
        return {"op": op, **_size(rng, 12, 160), "jitter": rng.random() < 0.5}
    if op == "jacobian":
        return {"op": op, **_size(rng, 12, 120), "jitter": rng.random() < 0.5}
    if op == "step":
        method = rng.choice(("plain", "two-level-fp16", "two-level-fp16", "two-level", "chebyshev", "bf16",
                             "matrix-free"))
        if method.startswith("two-level"):  # a coarse box grid wants sizes that it divides
            k = rng.randint(2, 10)
            size = {"nx": 10 * k, "ny": 10 * max(1, round(k / 2)), "nz": 10 * max(1, round(k / 2))}
        else:
            size = _size(rng, 12, 40)
        return {"op": op, "method": method, **size, "host": rng.random() < 0.3}
    if op == "filter":
        return {"op": op, **_size(rng, 16, 100), "length": round(rng.uniform(0.02, 0.2), 3)}
    if op == "batch":
        return {"op": op, "count": rng.randint(2, 12)}
    return {"op": op, "n0": rng.randint(17, 65), "n1": rng.randint(9, 33), "n2": rng.randint(9, 33),
            "batch": rng.randint(1, 8)}


# ---- inputs --------------------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _mesh(nx, ny, nz, jitter=False, seed=0):
    """Coordinates (N, 3) and connectivity (C, 4) on the GPU, and the loaded faces at x = 2 as
    (cells, local nodes) and the clamped nodes at x = 0."""
    n = (nx + 1, ny + 1, nz + 1)
    ax = [torch.arange(m, dtype=torch.float64, device="cuda") * (length / (m - 1)) for m, length in zip(n, (2.0, 1.0, 1.0))]
    x = torch.stack(torch.meshgrid(*ax, indexing="ij"), -1)
    if jitter:
        move = torch.rand(*n, 3, generator=_gen(seed), device="cuda", dtype=torch.float64) * 2 - 1
        spacing = torch.tensor([2.0 / nx, 1.0 / ny, 1.0 / nz], dtype=torch.float64, device="cuda")
        x[1:-1, 1:-1, 1:-1] += 0.15 * (move * spacing)[1:-1, 1:-1, 1:-1]
    ids = torch.arange(n[0] * n[1] * n[2], dtype=torch.int32, device="cuda").reshape(n)
    corner = lambda o: ids[o[0]:o[0] + nx, o[1]:o[1] + ny, o[2]:o[2] + nz].reshape(-1)  # noqa: E731
    tets = [torch.stack([corner((0, 0, 0)), corner(RING[t]), corner(RING[(t + 1) % 6]), corner((1, 1, 1))], -1)
            for t in range(6)]
    conn = torch.stack(tets, 1).reshape(-1, 4)
    on = ids[-1].reshape(-1).min() <= conn  # the x = 2 nodes are the last plane of the numbering
    cells = torch.nonzero(on.sum(1) == 3).reshape(-1)
    local = torch.nonzero(on[cells])[:, 1].reshape(-1, 3)
    return x.reshape(-1, 3).contiguous(), conn.contiguous(), (cells.int(), local.int()), ids[0].reshape(-1)


def _density(N, seed):
    """Nodal densities, independent and uniform in [0.01, 1], as the benchmark has them."""
    return torch.rand(N, generator=_gen(seed), device="cuda", dtype=torch.float64) * 0.99 + 0.01


def _smooth_density(n, rng):
    """A design-like density on (n+1)(n/2+1)^2 nodes: a Gaussian random field of correlation
    length 0.1 through the logistic function."""
    shape, lengths = (n + 1, n // 2 + 1, n // 2 + 1), (2.0, 1.0, 1.0)
    noise = torch.from_numpy(rng.standard_normal(shape)).cuda()
    k = torch.meshgrid(*[2 * math.pi * torch.fft.fftfreq(m, d=l / (m - 1), dtype=torch.float64, device="cuda")
                         for m, l in zip(shape, lengths)], indexing="ij")
    field = torch.fft.ifftn(torch.fft.fftn(noise) * torch.exp(-0.25 * (k[0] ** 2 + k[1] ** 2 + k[2] ** 2) * 0.01)).real
    return torch.sigmoid((field - field.mean()) / field.std()).clamp(0.01, 1.0).reshape(-1)


def _field(x, seed):
    """A displacement-like field: smooth waves of random phase and a small rough part."""
    g = _gen(seed)
    c = torch.rand(3, 8, generator=g, device="cuda", dtype=torch.float64)
    waves = [c[d, 0] * torch.sin(2 * c[d, 1] * x[:, 0] + c[d, 2]) * torch.cos(3 * c[d, 3] * x[:, 1] + c[d, 4])
             * torch.cos(3 * c[d, 5] * x[:, 2] + c[d, 6]) for d in range(3)]
    rough = torch.rand(x.shape[0], 3, generator=g, device="cuda", dtype=torch.float64) - 0.5
    return (torch.stack(waves, 1) + 1e-3 * rough).reshape(-1).contiguous()


def _elastic_inputs(case, seed):
    jitter = bool(case.get("jitter"))
    x, conn, load, clamped = _mesh(case["nx"], case["ny"], case["nz"], jitter, seed)
    u = _field(x, seed + 2)
    if case["op"] == "matrix_free":  # a Krylov vector: zero on the clamped face
        u.reshape(-1, 3)[clamped.long()] = 0.0
    return {"x": x, "conn": conn, "load": load, "clamped": clamped, "traction": (0.0, -1.0, 0.0),
            "z": _density(x.shape[0], seed + 1), "u": u, "lam": _field(x, seed + 3)}


def _batch_inputs(case, seed):
    """Cantilevers of n x n/2 x n/2 hexes, the n of the batch workload in turn, with a random
    design and load direction each."""
    rng, members = np.random.default_rng(seed), []
    for k in range(case["count"]):
        n = BATCH_SIZES[k % 5]
        x, conn, load, clamped = _mesh(n, n // 2, n // 2)
        d = rng.standard_normal(3)
        members.append({"x": x, "conn": conn, "load": load, "clamped": clamped,
                        "traction": tuple(float(v) for v in d / np.linalg.norm(d)), "z": _smooth_density(n, rng)})
    return members


def _network_inputs(case, seed):
    """He-normal parameters, the 8 features of designs (density, face masks, coordinates, the
    density cubed) and unit-RMS response fields as targets."""
    rng = np.random.default_rng(seed)
    parts = []
    for ci, co, taps in LAYERS:
        parts += [rng.standard_normal(taps * co * ci) * math.sqrt((2.0 if taps == 27 else 1.0) / (taps * ci)), np.zeros(co)]
    n, B, g = (case["n0"], case["n1"], case["n2"]), case["batch"], _gen(seed)
    pos = torch.stack(torch.meshgrid(*[torch.linspace(0, 1, m, device="cuda") for m in n], indexing="ij"), -1)
    feat = torch.zeros(B, *n, 8, device="cuda")
    feat[..., 0] = torch.sigmoid(torch.randn(B, *n, generator=g, device="cuda"))
    feat[:, -1, :, :, 1] = 1.0
    feat[:, 0, :, :, 2] = 1.0
    feat[..., 3:6] = pos
    feat[..., 6] = feat[..., 0] ** 3
    c = torch.rand(B, 1, 1, 1, 9, 3, generator=g, device="cuda")
    target = torch.sin(4 * (pos[None, :, :, :, None, :] * c).sum(-1) + 6 * c[..., 0])
    nodes = n[0] * n[1] * n[2]
    return np.concatenate(parts).astype(np.float32), feat.reshape(B, nodes, 8).contiguous(), target.reshape(B, nodes, 9).contiguous()


# ---- one pass ------------------------------------------------------------------------------


def _spec(m, solver=None):
    from platoanalyze_b200.problem import ProblemSpec, SolverOptions

    dofs = (3 * m["clamped"][:, None] + torch.arange(3, device="cuda")).reshape(-1).int().cpu().numpy()
    return ProblemSpec(m["x"].cpu().numpy(), m["conn"].cpu().numpy(), 1.0, NU, PENALTY, RHO_MIN,
                       [(m["load"][0].cpu().numpy(), m["load"][1].cpu().numpy(), m["traction"])],
                       dofs, np.zeros(dofs.size), solver or SolverOptions())


def prepare(case, seed):
    from platoanalyze_b200.learned import UNet
    from platoanalyze_b200.problem import EllipticProblem, HelmholtzFilter, SolverOptions
    from platoanalyze_b200.workloads import coarse_grid, method_options

    op = case["op"]
    if op in ("train", "forward"):
        params, inp, tgt = _network_inputs(case, seed)
        net = UNet((case["n0"], case["n1"], case["n2"]), case["batch"])
        net.set_params(params)
        return {"op": op, "net": net, "inp": inp, "tgt": tgt, "step": 0}
    if op == "filter":
        x, conn, _, _ = _mesh(case["nx"], case["ny"], case["nz"])
        flt = HelmholtzFilter(x.cpu().numpy(), conn.cpu().numpy(), case["length"])
        return {"op": op, "filter": flt, "z": _density(x.shape[0], seed + 1), "w": _density(x.shape[0], seed + 2) - 0.5}
    if op == "batch":
        members = _batch_inputs(case, seed)
        # the batch workload's method (Chebyshev(8)-Jacobi on an FP32 copy, FP64 outside)
        opts = method_options("chebyshev", 1e-10)
        prob = EllipticProblem.batch([_spec(m, opts) for m in members])
        return {"op": op, "problem": prob, "z": torch.cat([m["z"] for m in members])}
    m = _elastic_inputs(case, seed)
    opts = SolverOptions()
    if op == "step":
        opts = method_options(case["method"], 1e-10, coarse_grid(case["nx"], case["ny"], case["nz"]))
    prob = EllipticProblem(_spec(m, opts))
    state = {"op": op, "problem": prob, "z": m["z"], "u": m["u"], "lam": m["lam"]}
    if op == "step" and case["host"]:
        pinned = lambda n: torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()  # noqa: E731
        state |= {"z_host": pinned(m["z"].numel()), "u_host": pinned(m["u"].numel()), "g_host": pinned(m["z"].numel())}
        state["z_host"][:] = m["z"].cpu().numpy()
    return state


def run(s):
    op = s["op"]
    if op == "residual":
        return s["problem"].vf_value(s["u"], s["z"])
    if op == "jacobian":
        return s["problem"].vf_gradient_u(s["u"], s["z"])
    if op == "adjoint":
        p = s["problem"]
        g = p.sf_gradient_z(s["u"], s["z"])
        return p.sf_gradient_u(s["u"], s["z"]), p.vf_gradient_z_apply(s["u"], s["z"], s["lam"], g)
    if op == "criterion":
        return s["problem"].criterion_value_and_gradient(s["z"], s["u"])[:2]
    if op == "matrix_free":
        return s["problem"].apply_operator(s["z"], s["u"], 1)
    if op == "step":
        if "z_host" in s:
            return s["problem"].solve_and_gradient_host(s["z_host"], None, s["u_host"], s["g_host"])[:3]
        u, _ = s["problem"].solution(s["z"])
        return (u, *s["problem"].criterion_value_and_gradient(s["z"], u)[:2])
    if op == "filter":
        return s["filter"].solution(s["z"])[0], s["filter"].criterion_gradient(s["w"])[0]
    if op == "batch":
        u, _ = s["problem"].solution(s["z"])
        return u, s["problem"].batch_criterion_values(s["z"], u), s["problem"].criterion_gradient(s["z"], u)[0]
    if op == "forward":
        return s["net"].forward(s["inp"])
    s["step"] += 1
    loss, grads = s["net"].loss_and_gradients(s["inp"], s["tgt"], want_grads=True)
    s["net"].adam_step(1e-4, s["step"])
    return loss, grads


def _edges(a, b, c):
    """Edges of the mesh: along the axes, across the hex faces, through the hexes."""
    axes = a * (b + 1) * (c + 1) + (a + 1) * b * (c + 1) + (a + 1) * (b + 1) * c
    return axes + a * b * (c + 1) + a * (b + 1) * c + (a + 1) * b * c + a * b * c


def work(case):
    """Each input read once, each output written once, and the operations of the formulas; for
    the solves one build of the operator and one product with it, whatever the method."""
    op = case["op"]
    if op in ("train", "forward"):
        n = [(case[k] + 3) // 4 * 4 for k in ("n0", "n1", "n2")]
        level = [case["batch"] * n[0] * n[1] * n[2] // 8 ** k for k in range(3)]
        at = (0, 0, 1, 1, 2, 2, 1, 1, 0, 0, 0)
        flops = sum(2 * level[l] * ci * co * t for (ci, co, t), l in zip(LAYERS, at))
        nodes = case["batch"] * case["n0"] * case["n1"] * case["n2"]
        params = sum(ci * co * t + co for ci, co, t in LAYERS)
        if op == "forward":
            return {"bytes": 4 * (nodes * 17 + params), "flops": flops}
        return {"bytes": 4 * (nodes * 17 + 7 * params), "flops": 3 * flops}
    if op == "batch":
        sizes = [(n, n // 2, n // 2) for n in (BATCH_SIZES[k % 5] for k in range(case["count"]))]
    else:
        sizes = [(case["nx"], case["ny"], case["nz"])]
    N = sum((a + 1) * (b + 1) * (c + 1) for a, b, c in sizes)
    C = sum(6 * a * b * c for a, b, c in sizes)
    B = N + 2 * sum(_edges(*n) for n in sizes)
    mesh = 16 * C + 24 * N
    return {
        "residual": {"bytes": mesh + 8 * N + 72 * N, "flops": 260 * C},
        "jacobian": {"bytes": mesh + 8 * N + 4 * B + 4 * N + 72 * B, "flops": 500 * C},
        "adjoint": {"bytes": mesh + 8 * N + 80 * N, "flops": 400 * C},
        "criterion": {"bytes": mesh + 8 * N + 32 * N, "flops": 200 * C},
        "matrix_free": {"bytes": mesh + 8 * N + 48 * N, "flops": 260 * C},
        "step": {"bytes": mesh + 8 * N + 76 * B + 4 * N + 56 * N, "flops": 700 * C + 18 * B},
        "batch": {"bytes": mesh + 8 * N + 76 * B + 4 * N + 56 * N, "flops": 700 * C + 18 * B},
        "filter": {"bytes": mesh + 32 * N + 2 * 12 * B, "flops": 100 * C + 4 * B},
    }[op]


# ---- the results in 64 bits ------------------------------------------------------------------


def _geometry(x, conn):
    """Basis gradients (C, 4, 3) and volumes (C) of the cells."""
    v = x[conn.long()]
    J = (v[:, :3] - v[:, 3:4]).transpose(1, 2)  # J[d][a] = x_a - x_3
    c0, c1, c2 = J[:, :, 0], J[:, :, 1], J[:, :, 2]
    det = (c0 * torch.linalg.cross(c1, c2)).sum(1)
    rows = torch.stack([torch.linalg.cross(c1, c2), torch.linalg.cross(c2, c0), torch.linalg.cross(c0, c1)], 1) / det[:, None, None]
    return torch.cat([rows, -rows.sum(1, keepdim=True)], 1), det.abs() / 6


def _chunks(C, size=400_000):
    return [slice(k, min(C, k + size)) for k in range(0, C, size)]


def _strain(g, ue):
    H = torch.einsum("cai,caj->cij", ue, g)  # du_i / dx_j
    return 0.5 * (H + H.transpose(1, 2))


def _stress(E):
    tr = E.diagonal(dim1=1, dim2=2).sum(1)
    return LAMBDA * tr[:, None, None] * torch.eye(3, dtype=E.dtype, device=E.device) + 2 * MU * E


def _load(m):
    F = torch.zeros_like(m["x"])
    cells, local = m["load"][0].long(), m["load"][1].long()
    ids = m["conn"].long()[cells].gather(1, local)
    p = m["x"][ids]
    area = torch.linalg.cross(p[:, 0] - p[:, 2], p[:, 1] - p[:, 2]).norm(dim=1) / 2
    t = torch.tensor(m["traction"], dtype=torch.float64, device="cuda")
    for a in range(3):
        F.index_add_(0, ids[:, a], area[:, None] / 3 * t)
    return F


def _exact_pass(m, u, z, lam=None):
    """Internal force, energy, d energy / dz (u fixed) and (dR/dz)^T lambda on the mesh."""
    N, conn = m["x"].shape[0], m["conn"]
    f, dfdz, dl = torch.zeros(N, 3, dtype=torch.float64, device="cuda"), *(torch.zeros(N, dtype=torch.float64, device="cuda") for _ in range(2))
    energy = 0.0
    for c in _chunks(conn.shape[0]):
        ids = conn[c].long()
        g, vol = _geometry(m["x"], conn[c])
        E = _strain(g, u.reshape(-1, 3)[ids])
        S = _stress(E)
        rho = z[ids].mean(1)
        s, ds = RHO_MIN + (1 - RHO_MIN) * rho ** PENALTY, (1 - RHO_MIN) * PENALTY * rho ** (PENALTY - 1) / 4
        dens = (S * E).sum((1, 2))
        energy += float((0.5 * vol * s * dens).sum())
        fe = torch.einsum("cij,caj->cai", S, g) * (vol * s)[:, None, None]
        dlam = (S * _strain(g, lam.reshape(-1, 3)[ids])).sum((1, 2)) * vol * ds if lam is not None else None
        for a in range(4):
            f.index_add_(0, ids[:, a], fe[:, a])
            dfdz.index_add_(0, ids[:, a], 0.5 * vol * ds * dens)
            if lam is not None:
                dl.index_add_(0, ids[:, a], dlam)
    return f.reshape(-1), energy, dfdz, dl


def _pattern(conn, N):
    pairs = [torch.unique(conn[:, a].long() * N + conn[:, b].long()) for a in range(4) for b in range(4)]
    return torch.unique(torch.cat(pairs))


def _assemble(conn, N, keys, block):
    """Sum of block(cells slice) -> (n, 4, 4, k) values over the node pairs of `keys`."""
    out = None
    for c in _chunks(conn.shape[0]):
        v = block(c)
        if out is None:
            out = torch.zeros(keys.numel(), v.shape[-1], dtype=torch.float64, device="cuda")
        ids = conn[c].long()
        at = torch.searchsorted(keys, (ids[:, :, None] * N + ids[:, None, :]).reshape(-1))
        out.index_add_(0, at, v.reshape(-1, v.shape[-1]))
    return out


def _stiffness(m, z, keys):
    def block(c):
        g, vol = _geometry(m["x"], m["conn"][c])
        w = vol * (RHO_MIN + (1 - RHO_MIN) * z[m["conn"][c].long()].mean(1) ** PENALTY)
        gg = torch.einsum("cai,cbj->cabij", g, g) * w[:, None, None, None, None]
        tr = gg.diagonal(dim1=3, dim2=4).sum(-1)
        K = LAMBDA * gg + MU * gg.transpose(3, 4) + MU * tr[..., None, None] * torch.eye(3, dtype=torch.float64, device="cuda")
        return K.reshape(*K.shape[:3], 9)
    return _assemble(m["conn"], m["x"].shape[0], keys, block)


def _cg(A, d, b, tol, most):
    """Jacobi-preconditioned conjugate gradients on a CSR matrix."""
    x, r = torch.zeros_like(b), b.clone()
    z = r / d
    p, rz, stop = z.clone(), r @ z, tol * tol * (b @ b)
    for k in range(most):
        q = A @ p
        alpha = rz / (p @ q)
        x.add_(alpha * p)
        r.sub_(alpha * q)
        if k % 25 == 24 and float(r @ r) <= float(stop):
            break
        z = r / d
        new = r @ z
        p = z + (new / rz) * p
        rz = new
    return x


def _exact_state(m):
    """The displacement under the load: the constrained system by conjugate gradients."""
    N, z = m["x"].shape[0], m["z"]
    keys = _pattern(m["conn"], N)
    K = _stiffness(m, z, keys).reshape(-1, 3, 3)
    row, col = keys // N, keys % N
    free = torch.ones(N, dtype=torch.float64, device="cuda")
    free[m["clamped"].long()] = 0.0
    K *= (free[row] * free[col])[:, None, None]
    K[row == col] += (1 - free)[:, None, None] * torch.eye(3, dtype=torch.float64, device="cuda")
    diag = K[row == col].diagonal(dim1=1, dim2=2).reshape(-1)
    b = (_load(m) * free[:, None]).reshape(-1)
    count = torch.bincount(row, minlength=N)
    first = torch.cumsum(count, 0) - count
    # rows of scalars: each block row becomes three, its blocks' rows side by side
    n = count.repeat_interleave(3)
    crow = torch.zeros(3 * N + 1, dtype=torch.int64, device="cuda")
    crow[1:] = torch.cumsum(3 * n, 0)
    place = torch.arange(keys.numel(), device="cuda") - first[row]
    val = torch.empty(9 * keys.numel(), dtype=torch.float64, device="cuda")
    cols = torch.empty(9 * keys.numel(), dtype=torch.int32, device="cuda")
    for i in range(3):
        at = crow[3 * row + i] + 3 * place
        for j in range(3):
            val[at + j] = K[:, i, j]
            cols[at + j] = (3 * col + j).int()
    del K
    A = torch.sparse_csr_tensor(crow.int(), cols, val, size=(3 * N, 3 * N))
    return _cg(A, diag, b, 1e-13, 12000)


def _exact_filter(case, seed):
    x, conn, _, _ = _mesh(case["nx"], case["ny"], case["nz"])
    N = x.shape[0]
    keys = _pattern(conn, N)

    def block(c):
        g, vol = _geometry(x, conn[c])
        M = vol[:, None, None] / 16 * torch.ones(4, 4, dtype=torch.float64, device="cuda")
        return torch.stack([case["length"] ** 2 * vol[:, None, None] * (g @ g.transpose(1, 2)) + M, M], -1)

    KM = _assemble(conn, N, keys, block)
    row, col = keys // N, keys % N
    crow = torch.zeros(N + 1, dtype=torch.int64, device="cuda")
    crow[1:] = torch.cumsum(torch.bincount(row, minlength=N), 0)
    K, M = (torch.sparse_csr_tensor(crow, col, KM[:, k].contiguous(), size=(N, N)) for k in range(2))
    diag = KM[row == col, 0]
    control, w = _density(N, seed + 1), _density(N, seed + 2) - 0.5
    return _cg(K, diag, M @ control, 1e-15, 2000), M @ _cg(K, diag, w, 1e-15, 2000)


def _exact_network(case, seed):
    params, inp, tgt = _network_inputs(case, seed)
    n, B = (case["n0"], case["n1"], case["n2"]), case["batch"]
    flat = torch.from_numpy(params).cuda().double().requires_grad_(case["op"] == "train")
    g = [(v + 3) // 4 * 4 for v in n]
    layers, at = [], 0
    for ci, co, taps in LAYERS:
        layers.append((flat[at:at + taps * co * ci].reshape(taps, co, ci), flat[at + taps * co * ci:at + taps * co * ci + co]))
        at += taps * co * ci + co

    def conv(a, k, relu=True):
        w, b = layers[k]
        pad = torch.nn.functional.pad(a, (0, 0, 1, 1, 1, 1, 1, 1))
        D, H, W = a.shape[1:4]
        y = b + 0
        for t in range(w.shape[0]):
            dz, dy, dx = (t // 9, t // 3 % 3, t % 3) if w.shape[0] == 27 else (1, 1, 1)
            y = y + pad[:, dz:dz + D, dy:dy + H, dx:dx + W] @ w[t].T
        return y.relu() if relu else y

    def pool(a):
        return a.reshape(a.shape[0], a.shape[1] // 2, 2, a.shape[2] // 2, 2, a.shape[3] // 2, 2, a.shape[4]).mean((2, 4, 6))

    def up(a):
        return a.repeat_interleave(2, 1).repeat_interleave(2, 2).repeat_interleave(2, 3)

    def net(one):
        a = torch.zeros(1, *g, 16, dtype=torch.float64, device="cuda")
        a[:, :n[0], :n[1], :n[2], :8] = one.double().reshape(1, *n, 8)
        s0 = conv(conv(a, 0), 1)
        s1 = conv(conv(pool(s0), 2), 3)
        a = conv(conv(pool(s1), 4), 5)
        a = conv(conv(torch.cat([up(a), s1], -1), 6), 7)
        a = conv(conv(torch.cat([up(a), s0], -1), 8), 9)
        return conv(a, 10, False)[:, :n[0], :n[1], :n[2]].reshape(1, -1, 9)

    if case["op"] == "forward":
        with torch.no_grad():
            return torch.cat([net(inp[k]) for k in range(B)])
    total, grad = 0.0, torch.zeros_like(flat)
    for k in range(B):
        loss = ((net(inp[k]) - tgt[k].double()) ** 2).sum() / tgt.numel()
        # the layers' views of the parameters are shared by the members
        grad += torch.autograd.grad(loss, flat, retain_graph=True)[0]
        total += float(loss.detach())
        del loss
    return total, grad


def exact(case, seed):
    op = case["op"]
    if op in ("train", "forward"):
        return _exact_network(case, seed)
    if op == "filter":
        return _exact_filter(case, seed)
    if op == "batch":
        us, vs, gs = [], [], []
        for m in _batch_inputs(case, seed):
            u = _exact_state(m)
            _, v, g, _ = _exact_pass(m, u, m["z"])
            us.append(u), vs.append(v), gs.append(-g)
        return torch.cat(us), np.array(vs), torch.cat(gs)
    m = _elastic_inputs(case, seed)
    if op == "jacobian":
        return _stiffness(m, m["z"], _pattern(m["conn"], m["x"].shape[0])).reshape(-1)
    if op == "step":
        u = _exact_state(m)
        _, v, g, _ = _exact_pass(m, u, m["z"])
        return u, v, -g
    u = m["u"]
    if op == "matrix_free":
        f = _exact_pass(m, u, m["z"])[0].reshape(-1, 3)
        f[m["clamped"].long()] = 0.0
        return f.reshape(-1)
    f, v, g, dl = _exact_pass(m, u, m["z"], m["lam"] if op == "adjoint" else None)
    if op == "residual":
        return f - _load(m).reshape(-1)
    return (f, g + dl) if op == "adjoint" else (v, -g)
