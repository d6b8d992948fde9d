"""The work that users of this library have it do, as measurable cases.

Every case goes through the public Python interface (`seldon_b200.api`,
`seldon_b200.autograd`).  `listed()` holds the named workloads, `draw(rng)`
gives others of the same ranges: products with a matrix, Krylov solves with
each kind of preconditioner, the preconditioner applies themselves,
mixed-precision and batched solves, a differentiated solve and the assembly
of a matrix.

Right-hand sides are made from a chosen solution x*, b = A x*, so `exact`
knows the answer of a solve without solving.  Solves run to a relative
residual of 1e-13, near what doubles can carry, so that the solution does not
depend on the step at which the test happens to stop.
"""
import math

import numpy as np
import torch

from seldon_b200 import api, autograd, matgen

TOL = 1e-13


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # one product with a small matrix: the call itself is what costs
        {"name": "mlt_lap2d_100", "op": "mlt", "matrix": "lap2d", "g": 100, "storage": "sym", "trans": False},
        # the product that a large solve repeats
        {"name": "mlt_convdiff_128", "op": "mlt", "matrix": "convdiff", "g": 128, "storage": "general",
         "trans": False},
        # rows of very uneven length (power law), columns all over x
        {"name": "mlt_zipf_500k", "op": "mlt", "matrix": "zipf", "g": 500000, "storage": "general",
         "trans": False},
        # a small symmetric system, the size of Seldon's own examples
        {"name": "cg_lap2d_100", "op": "solve", "solver": "cg", "matrix": "lap2d", "g": 100, "storage": "sym",
         "precond": "identity", "restart": 10},
        # a middle-sized nonsymmetric system
        {"name": "bicgstab_convdiff_80", "op": "solve", "solver": "bicgstab", "matrix": "convdiff", "g": 80,
         "storage": "general", "precond": "jacobi", "restart": 10},
        # a large nonsymmetric system with the reference's usual solver
        {"name": "gmres30_convdiff_128", "op": "solve", "solver": "gmres", "matrix": "convdiff", "g": 128,
         "storage": "general", "precond": "jacobi", "restart": 30},
        # the reference's own preconditioner in a symmetric solve
        {"name": "ssor_cg_poisson_64", "op": "solve", "solver": "cg", "matrix": "poisson", "g": 64,
         "storage": "sym", "precond": "sor", "restart": 10},
        # one application of an incomplete factor, as every step of a solver makes
        {"name": "ilu0_apply_convdiff_96", "op": "ilu0", "matrix": "convdiff", "g": 96, "trans": False},
        # a large symmetric system in mixed precision
        {"name": "ir_cg_poisson_160", "op": "ir", "solver": "cg", "matrix": "poisson", "g": 160,
         "restart": 30},
        # hundreds of uneven independent systems at once, with a tuned plan
        {"name": "batch_mixed_512", "op": "batch", "nsys": 512, "lo": 8, "hi": 140, "mixed": True,
         "tuned": True},
        # a solve and its gradients for every conductivity and for b
        {"name": "adjoint_graph_512", "op": "adjoint", "g": 512},
        # a matrix assembled from shuffled triplets
        {"name": "assemble_convdiff_128", "op": "assemble", "matrix": "convdiff", "g": 128, "shuffled": True,
         "symmetric": False},
    ]


def draw(rng):
    """One more case: the operations of `listed()` over the sizes they are used at."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["mlt", "mlt", "mlt", "solve", "solve", "solve", "sor", "ilu0", "ir", "batch", "adjoint",
                     "assemble"])
    if op == "mlt":
        matrix = rng.choice(["lap2d", "poisson", "convdiff", "zipf"])
        g = {"lap2d": size(10, 1400), "poisson": size(5, 128), "convdiff": size(5, 128),
             "zipf": size(2000, 500000)}[matrix]
        storage = rng.choice(["sym", "general"]) if matrix in ("lap2d", "poisson") else "general"
        return {"op": "mlt", "matrix": matrix, "g": g, "storage": storage, "trans": rng.random() < 0.3}
    if op == "solve":
        solver = rng.choice(["cg", "bicgstab", "gmres"])
        if solver == "cg":
            matrix = rng.choice(["lap2d", "poisson"])
            g = size(10, 500) if matrix == "lap2d" else size(6, 128)
            storage = rng.choice(["sym", "general"])
        else:
            matrix, storage = "convdiff", "general"
            g = size(6, 128) if solver == "bicgstab" else size(6, 104)
        return {"op": "solve", "solver": solver, "matrix": matrix, "g": g, "storage": storage,
                "precond": rng.choice(["identity", "jacobi"]), "restart": rng.randint(20, 30)}
    if op == "sor":
        solver = rng.choice(["cg", "gmres"])
        matrix = "poisson" if solver == "cg" else "convdiff"
        storage = rng.choice(["sym", "general"]) if solver == "cg" else "general"
        return {"op": "solve", "solver": solver, "matrix": matrix, "g": size(8, 64), "storage": storage,
                "precond": "sor", "restart": rng.randint(10, 30)}
    if op == "ilu0":
        return {"op": "ilu0", "matrix": rng.choice(["poisson", "convdiff"]), "g": size(8, 96),
                "trans": rng.random() < 0.3}
    if op == "ir":
        solver = rng.choice(["cg", "gmres"])
        return {"op": "ir", "solver": solver, "matrix": "poisson" if solver == "cg" else "convdiff",
                "g": size(24, 160 if solver == "cg" else 96), "restart": rng.randint(20, 30)}
    if op == "batch":
        lo = size(4, 40)
        return {"op": "batch", "nsys": size(16, 512), "lo": lo, "hi": rng.randint(lo + 1, 140),
                "mixed": rng.random() < 0.7, "tuned": rng.random() < 0.5}
    if op == "adjoint":
        return {"op": "adjoint", "g": size(16, 512)}
    matrix = rng.choice(["lap2d", "poisson", "convdiff", "zipf"])
    g = {"lap2d": size(10, 1400), "poisson": size(5, 128), "convdiff": size(5, 128),
         "zipf": size(2000, 200000)}[matrix]
    return {"op": "assemble", "matrix": matrix, "g": g, "shuffled": rng.random() < 0.7,
            "symmetric": rng.random() < 0.3}


# ------------------------------------------------------------------ matrices

def _rng(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _stencil(matrix, g):
    """(dims, [(offset, value)], diagonal) of a grid operator."""
    if matrix == "lap2d":
        return (g, g, 1), [((-1, 0, 0), -1.0), ((1, 0, 0), -1.0), ((0, -1, 0), -1.0), ((0, 1, 0), -1.0)], 4.0
    if matrix == "poisson":
        return (g, g, g), [(o, -1.0) for o in ((-1, 0, 0), (1, 0, 0), (0, -1, 0), (0, 1, 0), (0, 0, -1),
                                               (0, 0, 1))], 6.0
    # first-order upwind convection-diffusion, velocity (1, 0.5, 0.25), Peclet 10
    v = (1.0, 0.5, 0.25)
    eps, h = math.sqrt(sum(t * t for t in v)) / 10.0, 1.0 / (g + 1)
    off = []
    for d in range(3):
        for side in (-1, 1):
            o = [0, 0, 0]
            o[d] = side
            off.append((tuple(o), -eps - (h * v[d] if side < 0 else 0.0)))
    return (g, g, g), off, 6.0 * eps + h * sum(v)


def _grid(dims):
    gx, gy, gz = dims
    i = torch.arange(gx * gy * gz, device="cuda")
    return i, i % gx, (i // gx) % gy, i // (gx * gy)


def _inside(dims, ix, iy, iz, o):
    gx, gy, gz = dims
    x, y, z = ix + o[0], iy + o[1], iz + o[2]
    return (x >= 0) & (x < gx) & (y >= 0) & (y < gy) & (z >= 0) & (z < gz)


def _stencil_triplets(matrix, g, upper=False):
    """Row, column and value of every entry of a grid operator, in row order."""
    dims, off, diag = _stencil(matrix, g)
    i, ix, iy, iz = _grid(dims)
    step = lambda o: o[0] + o[1] * dims[0] + o[2] * dims[0] * dims[1]  # noqa: E731
    every = sorted([((0, 0, 0), diag)] + off, key=lambda e: step(e[0]))
    if upper:
        every = [e for e in every if step(e[0]) >= 0]
    ok = torch.stack([_inside(dims, ix, iy, iz, o) for o, _ in every], 1)
    col = torch.stack([i + step(o) for o, _ in every], 1)
    val = torch.tensor([c for _, c in every], dtype=torch.float64, device="cuda").expand(i.numel(), -1)
    row = i[:, None].expand(-1, len(every))
    return row[ok].int(), col[ok].int(), val[ok]


def _zipf_triplets(n, seed):
    """Rows of Zipf(1.5) length clipped to [1, 2000], columns anywhere, a
    dominant diagonal; in row and column order."""
    gen = _rng(seed)
    k = torch.arange(1, 2001, device="cuda", dtype=torch.float64)
    p = k ** -1.5
    p[-1] = 2.0 * 2000.0 ** -0.5  # all the longer ones
    lens = torch.multinomial(p, n, replacement=True, generator=gen) + 1
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), lens)
    cols = torch.randint(0, n, (rows.numel(),), device="cuda", generator=gen)
    keys = torch.unique(torch.cat([rows * n + cols, torch.arange(n, device="cuda") * (n + 1)]))
    r, c = keys // n, keys % n
    v = torch.randn(r.numel(), dtype=torch.float64, device="cuda", generator=gen)
    absolute = torch.zeros(n, dtype=torch.float64).index_add_(0, r.cpu(), v.abs().cpu()).cuda()
    v = torch.where(r == c, 1.0 + absolute[r], v)
    return r.int(), c.int(), v


def _triplets(case, seed, upper=False):
    if case["matrix"] == "zipf":
        return _zipf_triplets(case["g"], seed)
    return _stencil_triplets(case["matrix"], case["g"], upper)


def _order(case):
    g = case["g"]
    return {"lap2d": g * g, "poisson": g ** 3, "convdiff": g ** 3, "zipf": g}[case["matrix"]]


def _nnz(case):
    g = case["g"]
    return {"lap2d": 5 * g * g - 4 * g, "poisson": 7 * g ** 3 - 6 * g * g, "convdiff": 7 * g ** 3 - 6 * g * g,
            "zipf": 68 * g}[case["matrix"]]


def _matrix(case, seed):
    n = _order(case)
    sym = case.get("storage") == "sym"
    r, c, v = _triplets(case, seed, upper=sym)
    ptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.cumsum(torch.bincount(r.long(), minlength=n), 0)
    arrays = (ptr.int().cpu().numpy(), c.cpu().numpy(), v.cpu().numpy())
    return api.RowSymSparse(n, *arrays) if sym else api.RowSparse(n, n, *arrays)


def _stencil_times(matrix, g, x, trans=False):
    """A x by shifts of the grid: the same bits on every run."""
    dims, off, diag = _stencil(matrix, g)
    gx, gy, gz = dims
    u = x.view(gz, gy, gx)
    y = diag * u

    def ends(n, s):
        return (slice(None), slice(None)) if s == 0 else \
            ((slice(0, n - 1), slice(1, n)) if s > 0 else (slice(1, n), slice(0, n - 1)))

    for o, c in off:
        o = tuple(-t for t in o) if trans else o
        (zt, zf), (yt, yf), (xt, xf) = ends(gz, o[2]), ends(gy, o[1]), ends(gx, o[0])
        y[zt, yt, xt] += c * u[zf, yf, xf]
    return y.reshape(-1)


def _solution(case, seed):
    return torch.rand(_order(case), dtype=torch.float64, device="cuda", generator=_rng(seed + 7919)) * 2 - 1


def _batch_sides(case):
    """The systems' sizes are the case's own; their solutions come from the seed."""
    return np.random.default_rng(case["nsys"]).integers(case["lo"], case["hi"] + 1, case["nsys"])


def _batch_solution(case, seed):
    n = int((_batch_sides(case).astype(np.int64) ** 2).sum())
    return np.random.default_rng(seed + 7919).uniform(-1, 1, n)


def _adjoint_inputs(case, seed):
    """Conductivities, the solution x* and the adjoint solution of a grid."""
    g, gen = case["g"], _rng(seed)
    n = g * g
    idx = torch.arange(n, device="cuda").view(g, g)
    edges = torch.cat([torch.stack([idx[:, :-1].reshape(-1), idx[:, 1:].reshape(-1)], 1),
                       torch.stack([idx[:-1, :].reshape(-1), idx[1:, :].reshape(-1)], 1)])
    theta = torch.randn(edges.shape[0], dtype=torch.float64, device="cuda", generator=gen).exp()
    xs = torch.rand(n, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1
    lam = torch.randn(n, dtype=torch.float64, device="cuda", generator=gen)
    return edges, theta, xs, lam


def _graph_times(g, theta, u, shift=1e-3):
    """(L(theta) + shift I) u on the g x g grid graph, by shifts."""
    w, n1 = u.view(g, g), g * (g - 1)
    th, tv = theta[:n1].view(g, g - 1), theta[n1:].view(g - 1, g)
    y = shift * w
    fh, fv = th * (w[:, :-1] - w[:, 1:]), tv * (w[:-1, :] - w[1:, :])
    y[:, :-1] += fh
    y[:, 1:] -= fh
    y[:-1, :] += fv
    y[1:, :] -= fv
    return y.reshape(-1)


# ------------------------------------------------------------------ what a program has in hand

def prepare(case, seed):
    op = case["op"]
    state = {"case": case}
    if op == "mlt":
        state["A"] = _matrix(case, seed)
        state["x"] = torch.randn(_order(case), dtype=torch.float64, device="cuda", generator=_rng(seed + 7919))
        state["y"] = torch.zeros(_order(case), dtype=torch.float64, device="cuda")
    elif op in ("solve", "ilu0", "ir"):
        A = _matrix(case, seed)
        state["A"] = A
        state["b"] = _stencil_times(case["matrix"], case["g"], _solution(case, seed))
        state["x"] = torch.zeros_like(state["b"])
        if op == "ilu0":
            M = api.IlutPreconditioning()
            M.SetFactorisationType(M.ILU_0)
            M.FactorizeMatrix(A)
            M.Solve(A, state["b"], state["x"])
        elif op == "ir":
            M = api.JacobiPreconditioner() if case["solver"] == "gmres" else None
        else:
            M = {"identity": api.Preconditioner_Base, "jacobi": api.JacobiPreconditioner,
                 "sor": api.SorPreconditioner}[case["precond"]]()
            if case["precond"] == "sor":
                M.Solve(A, state["b"], state["x"])
        state["M"] = M
    elif op == "batch":
        systems = [matgen.lap2d(int(s), shift=0.01) for s in _batch_sides(case)]
        xs = _batch_solution(case, seed)
        B = api.Batch(systems)
        b, at = [], 0
        for s in systems:
            n = len(s[0]) - 1
            b.append(matgen.matvec(*s, xs[at:at + n]))
            at += n
        state["B"] = B
        state["b"] = torch.from_numpy(np.concatenate(b)).cuda()
        state["x"] = torch.zeros_like(state["b"])
        if case["tuned"]:
            B.autotune(state["x"], state["b"], tol=TOL, mixed=case["mixed"])
    elif op == "adjoint":
        edges, theta, xs, lam = _adjoint_inputs(case, seed)
        state["lap"] = autograd.GraphLaplacian(case["g"] ** 2, edges.cpu().numpy(), 1e-3)
        state["theta"] = theta.requires_grad_()
        state["b"] = _graph_times(case["g"], theta.detach(), xs).requires_grad_()
        state["gx"] = _graph_times(case["g"], theta.detach(), lam)
    else:
        r, c, v = _triplets(case, seed)
        if case["matrix"] != "zipf":
            v = torch.randn(v.shape, dtype=torch.float64, device="cuda", generator=_rng(seed + 7919))
        if case["shuffled"]:
            at = torch.randperm(r.numel(), device="cuda", generator=_rng(seed + 104729))
            r, c, v = r[at], c[at], v[at]
        state["triplets"] = (r.contiguous(), c.contiguous(), v.contiguous())
    return state


# ------------------------------------------------------------------ one pass

def _iteration(case):
    it = api.Iteration(20000, TOL)
    it.SetRestart(case["restart"])
    it.HideMessages()
    return it


def run(state):
    case = state["case"]
    op = case["op"]
    if op == "mlt":
        api.Mlt(state["A"], state["x"], state["y"],
                trans=api.SeldonTrans if case["trans"] else api.SeldonNoTrans)
        return {"y": state["y"]}
    if op == "solve":
        solver = {"cg": api.Cg, "bicgstab": api.BiCgStab, "gmres": api.Gmres}[case["solver"]]
        code = solver(state["A"], state["x"], state["b"], state["M"], _iteration(case))
        return {"x": state["x"], "code": code}
    if op == "ilu0":
        M = state["M"]
        (M.TransSolve if case["trans"] else M.Solve)(state["A"], state["b"], state["x"])
        return {"x": state["x"]}
    if op == "ir":
        code, _ = api.IterativeRefinement(state["A"], state["x"], state["b"], state["M"], tol=TOL,
                                          solver=case["solver"], restart=case["restart"])
        return {"x": state["x"], "code": code}
    if op == "batch":
        state["B"].solve(state["x"], state["b"], summary=False, tol=TOL, mixed=case["mixed"])
        return {"x": state["x"]}
    if op == "adjoint":
        x = autograd.graph_laplacian_solve(state["theta"], state["b"], state["lap"], TOL)
        dtheta, db = torch.autograd.grad(x, (state["theta"], state["b"]), state["gx"])
        return {"x": x, "dtheta": dtheta, "db": db}
    m, n, ptr, ind, val = api.ConvertMatrix_from_Coordinates(*state["triplets"], symmetric=case["symmetric"])
    return {"m": m, "n": n, "ptr": ptr, "ind": ind, "val": val}


# ------------------------------------------------------------------ the least work

def _steps(case):
    """About how many steps a solve takes (measured on these operators)."""
    g = case["g"]
    if case.get("precond") == "sor":
        return 1.2 * g
    if case["matrix"] == "convdiff":
        return 5.0 * g if case["solver"] == "bicgstab" else 8.0 * g
    return 4.3 * g if case["matrix"] == "poisson" else 3.8 * g


def work(case):
    op = case["op"]
    if op == "batch":
        rows = case["nsys"] * (case["lo"] ** 2 + case["lo"] * case["hi"] + case["hi"] ** 2) / 3.0
        steps = 150.0
        return {"bytes": rows * (5 * 12 + 4 + 16), "flops": rows * steps * (2 * 5 + 10)}
    if op == "adjoint":
        n, steps = case["g"] ** 2, 2 * 6.0 * case["g"]
        return {"bytes": n * (5 * 12 + 4 + 10 * 8), "flops": n * steps * (2 * 5 + 10)}
    n, nnz = _order(case), _nnz(case)
    once = 12 * nnz + 4 * n + 16 * n
    if op == "mlt":
        return {"bytes": once, "flops": 2 * nnz}
    if op == "ilu0":
        return {"bytes": once, "flops": 2 * nnz + n}
    if op == "assemble":
        return {"bytes": 28 * nnz + 4 * n, "flops": 0}
    # a solve: its matrix and vectors once a step where they are larger than
    # the 126 MB cache, once in all where they are not
    steps = _steps(case)
    value = 4 if op == "ir" else 8
    vectors = {"cg": 8, "bicgstab": 10, "gmres": 2 + case["restart"] / 2}[case["solver"]]
    step = nnz * (value + 4) + n * value * vectors
    return {"bytes": step * (steps if step > 126e6 else 1), "flops": steps * (2 * nnz + 2 * vectors * n)}


# ------------------------------------------------------------------ the answers

def _ilu0_exact(case, seed):
    """ILU(0) of a grid operator and its two sweeps, one diagonal plane of the
    grid at a time.  Off the diagonal the factor keeps the operator's entries
    (no two neighbours of a point are neighbours of each other)."""
    dims, off, diag = _stencil(case["matrix"], case["g"])
    i, ix, iy, iz = _grid(dims)
    b = _stencil_times(case["matrix"], case["g"], _solution(case, seed))
    value = dict(off)
    steps = [(o, o[0] + o[1] * dims[0] + o[2] * dims[0] * dims[1]) for o, _ in off]
    level = ix + iy + iz
    order = torch.argsort(level, stable=True)
    planes = torch.split(order, torch.bincount(level).tolist())
    d = torch.full_like(b, diag)
    neighbours = []
    for rows in planes:
        x, y, z = ix[rows], iy[rows], iz[rows]
        near = []
        for o, s in steps:
            ok = _inside(dims, x, y, z, o)
            near.append((o, s, ok, torch.where(ok, rows + s, rows)))
        neighbours.append(near)

    def mirror(o):
        return tuple(-t for t in o)

    for rows, near in zip(planes, neighbours):
        for o, s, ok, at in near:
            if s < 0:
                d[rows] -= torch.where(ok, value[o] * value[mirror(o)] / d[at], torch.zeros_like(d[rows]))
    x = b.clone()

    def sweep(forward, unit, trans):
        for k in range(len(planes)) if forward else range(len(planes) - 1, -1, -1):
            rows = planes[k]
            t = x[rows].clone()
            for o, s, ok, at in neighbours[k]:
                if (s < 0) == forward:
                    c = value[mirror(o)] if trans else value[o]
                    # L = (strictly lower part) D^-1 has unit diagonal, U = D + (strictly upper part)
                    w = c / (d[rows] if trans else d[at]) if unit else c
                    t -= torch.where(ok, w * x[at], torch.zeros_like(t))
            x[rows] = t if unit else t / d[rows]

    if case["trans"]:
        sweep(True, False, True)
        sweep(False, True, True)
    else:
        sweep(True, True, False)
        sweep(False, False, False)
    return x


def exact(case, seed):
    op = case["op"]
    if op == "mlt":
        x = torch.randn(_order(case), dtype=torch.float64, device="cuda", generator=_rng(seed + 7919))
        if case["matrix"] != "zipf":
            return {"y": _stencil_times(case["matrix"], case["g"], x, case["trans"])}
        r, c, v = (t.cpu() for t in _zipf_triplets(case["g"], seed))
        r, c = (c, r) if case["trans"] else (r, c)
        y = torch.zeros(case["g"], dtype=torch.float64)
        return {"y": y.index_add_(0, r.long(), v * x.cpu()[c.long()])}
    if op in ("solve", "ir"):
        return {"x": _solution(case, seed), "code": None}
    if op == "ilu0":
        return {"x": _ilu0_exact(case, seed)}
    if op == "batch":
        return {"x": torch.from_numpy(_batch_solution(case, seed))}
    if op == "adjoint":
        edges, theta, xs, lam = _adjoint_inputs(case, seed)
        i, j = edges[:, 0], edges[:, 1]
        return {"x": xs, "dtheta": -(lam[i] - lam[j]) * (xs[i] - xs[j]), "db": lam}
    r, c, v = prepare(case, seed)["triplets"]
    if case["symmetric"]:
        keep = r <= c
        r, c, v = r[keep], c[keep], v[keep]
    at = torch.sort(r.long() * (int(c.max()) + 1) + c.long(), stable=True).indices
    return {"m": None, "n": None, "ptr": None, "ind": None, "val": v[at]}
