"""The work that users of the solver have it do, as timed cases.

Each case is one pass through the public binding (kinterp, ki_autograd): a
boundary factored and solved from host arrays, by the direct FP64 method or
by the refined mixed method; many boundaries factored together; a moving
boundary followed; a kept factorization solving new right-hand sides; the
operator applied; the solution summed on a grid; gradients with respect to
the boundary.  Sizes run from the ellipse of the smoke test (1,024 dofs) to
the Stokes disk with holes (65,536 dofs) and the batch of 256 stars
(about 800,000 dofs), odd sizes among them.
"""
import math
import os
import sys
import types

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "kern-interp-old_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import ki_autograd  # noqa: E402
import ki_geometry as G  # noqa: E402
import kinterp  # noqa: E402

LAPLACE, STOKES = 0, 2
REFINE_TOL = 1e-12


def listed():
    return [
        # the smallest whole call: one small boundary factored, solved and
        # evaluated at interior points from host arrays
        {"name": "laplace_1k_direct", "kind": "direct", "shape": "ellipse", "n": 1024,
         "leaf": 64},
        # an ordinary single problem by the reference's own method
        {"name": "laplace_16k_direct", "kind": "direct", "shape": "star", "n": 16384, "leaf": 64},
        # the same boundary by the mixed method
        {"name": "laplace_16k_refined", "kind": "refined", "shape": "star", "n": 16384,
         "leaf": 64, "id_tol": 3e-7},
        # the largest single problem, multiply connected, both methods
        {"name": "stokes_65k_direct", "kind": "direct", "shape": "stokes", "n": 32768,
         "holes": 8, "leaf": 64},
        {"name": "stokes_65k_refined", "kind": "refined", "shape": "stokes", "n": 32768,
         "holes": 8, "leaf": 64, "id_tol": 3e-8},
        # factor, solve and evaluate on a grid in one call, Laplace with
        # holes, node counts that divide into nothing, small leaves
        {"name": "annulus_grid", "kind": "integral", "n": 3001, "grid": 53, "leaf": 32},
        # many problems of uneven size in one factorization
        {"name": "batch_256", "kind": "batch", "count": 256, "nmin": 512, "nmax": 8192,
         "leaf": 64, "id_tol": 3e-7},
        # a moving boundary: two frames of a shape loop, each updated and solved
        {"name": "update_16k", "kind": "update", "n": 16384, "width": 0.03, "extra": 10,
         "leaf": 64},
        # shape gradients: forward solve, target potentials, backward
        {"name": "adjoint_8k", "kind": "adjoint", "n": 8192, "targets": 64, "leaf": 64},
        # a kept factorization, a new right-hand side (time stepping, the
        # preconditioner inside a caller's own iteration)
        {"name": "solve_stokes_65k", "kind": "solve", "shape": "stokes", "n": 32768, "holes": 8,
         "leaf": 64},
        # the operator with on-the-fly entries (a caller's own GMRES, residuals)
        {"name": "operator_stokes_65k", "kind": "operator", "shape": "stokes", "n": 32768,
         "holes": 8, "leaf": 64},
        # the potential on a grid of domain points from a known density
        {"name": "grid_350_star_16k", "kind": "grid", "n": 16384, "grid": 350, "leaf": 64},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["direct", "direct", "refined", "refined", "integral", "batch", "update",
                       "adjoint", "solve", "operator", "grid"])
    c = {"kind": kind, "leaf": rng.choice([32, 48, 64])}
    if kind in ("direct", "refined", "solve", "operator"):
        c["shape"] = rng.choice(["ellipse", "star", "stokes"])
        if c["shape"] == "stokes":
            c["n"] = _log_int(rng, 1024, 32768)
            c["holes"] = rng.randint(1, 8)
        else:
            c["n"] = _log_int(rng, 512, 16384)
        if kind == "refined":
            c["id_tol"] = 3e-8 if c["shape"] == "stokes" else 3e-7
    elif kind == "integral":
        c["n"], c["grid"] = _log_int(rng, 500, 6000), _log_int(rng, 16, 120)
    elif kind == "batch":
        c["count"] = _log_int(rng, 4, 200)
        c["nmin"], c["nmax"], c["id_tol"] = 512, _log_int(rng, 1024, 8192), 3e-7
    elif kind == "update":
        c["n"] = _log_int(rng, 2048, 16384)
        c["width"], c["extra"] = round(rng.uniform(0.03, 0.15), 3), rng.randint(-20, 40)
    elif kind == "adjoint":
        c["n"], c["targets"] = _log_int(rng, 1024, 8192), _log_int(rng, 8, 128)
    else:
        c["n"], c["grid"] = _log_int(rng, 1024, 16384), _log_int(rng, 24, 350)
    return c


# ---------------------------------------------------------------- problems
def _problem(case, seed):
    n, leaf = case["n"], case["leaf"]
    if case["shape"] == "ellipse":
        return G.ellipse_case(n=n, seed=seed, leaf_points=leaf)
    if case["shape"] == "star":
        return G.star_case(n=n, seed=seed, leaf_points=leaf)
    return G.stokes_holes_case(n_total=n, seed=seed, n_holes=case["holes"], leaf_points=leaf)


def _stars(case, seed):
    """Random stars whose sizes, log-uniform, belong to the case and whose
    shapes and data to the seed."""
    rng = np.random.default_rng(case["count"])
    sizes = np.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"]), case["count"]))
    rng = np.random.default_rng(seed)
    return [G.random_star(rng, int(n), case["leaf"]) for n in np.round(sizes)]


def _annulus(case, seed):
    """Laplace outside two holes: the data of four sources outside the disk."""
    pts, nrm, kap, w, holes = G.reference_shape("annulus", case["n"])
    rng = np.random.default_rng(seed)
    src, q = G.laplace_sources(rng, 4, 3.0)
    f = G.laplace_potential(pts, src, q)
    return G.Problem("annulus", LAPLACE, pts, nrm, kap, w, holes, f, np.zeros(0), np.zeros(0),
                     case["leaf"], 1e-10)


def _annulus_points(case):
    """A grid over the disk's square (x in the outer loop)."""
    g = np.linspace(-0.5, 1.5, case["grid"])
    return np.stack(np.meshgrid(g, g, indexing="ij"), 2).reshape(-1)


def _frames(case, seed):
    """The star and two later frames: a bump that appears and moves on."""
    rng = np.random.default_rng(seed)
    kw = dict(n=case["n"], leaf_points=case["leaf"], seed=seed, width=case["width"])
    c = rng.uniform(1.0, 4.0)
    return (G.star_case(n=case["n"], seed=seed, leaf_points=case["leaf"]),
            [G.bumped_star_case(center=c, amp=0.02, extra=case["extra"], **kw),
             G.bumped_star_case(center=c + 1.0, amp=0.03, extra=0, **kw)])


def _density(n, seed):
    """A smooth density on the star's nodes."""
    rng = np.random.default_rng(seed)
    t = 2.0 * np.pi * np.arange(n) / n
    mu = np.full(n, rng.standard_normal())
    for k in range(1, 9):
        a, b = rng.standard_normal(2) / k
        mu += a * np.cos(k * t) + b * np.sin(k * t)
    return mu


def _star_points(case):
    g = np.linspace(-1.3, 1.3, case["grid"])
    return np.stack(np.meshgrid(g, g, indexing="ij"), 2).reshape(-1)


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def _adjoint_inputs(case, seed):
    pr = G.fourier_star_case(n=case["n"], seed=seed, n_targets=case["targets"])
    return pr, [_dev(a) for a in (pr.points, pr.normals, pr.curvatures, pr.weights, pr.f)]


# ------------------------------------------------------------ prepare, run
def prepare(case, seed):
    kind = case["kind"]
    st = types.SimpleNamespace(case=case, kind=kind)
    if kind in ("direct", "refined"):
        st.pr = _problem(case, seed)
    elif kind == "integral":
        st.pr, st.pts = _annulus(case, seed), _annulus_points(case)
    elif kind == "batch":
        st.prs = _stars(case, seed)
        st.f = np.concatenate([p.f for p in st.prs])
    elif kind == "update":
        base, st.frames = _frames(case, seed)
        st.solver = kinterp.Solver(base)
    elif kind == "adjoint":
        st.pr, st.leaves = _adjoint_inputs(case, seed)
        for a in st.leaves:
            a.requires_grad_(True)
        st.targets, st.u_star = _dev(st.pr.targets), _dev(st.pr.extra["u_star"])
    else:
        # a kept factorization on a stream of the caller's
        st.pr = (G.star_case(n=case["n"], seed=seed, leaf_points=case["leaf"])
                 if kind == "grid" else _problem(case, seed))
        st.stream = torch.cuda.Stream()
        st.solver = kinterp.Solver(st.pr, stream=st.stream.cuda_stream)
        n, nb = st.solver.n_dofs, st.solver.n_border
        if kind == "solve":
            st.f = _dev(st.pr.f)
            st.z = torch.empty(n + nb, dtype=torch.float64, device="cuda")
            st.mu, st.alpha = st.z[:n], st.z[n:]
        elif kind == "operator":
            rng = np.random.default_rng(seed)
            st.x = _dev(rng.standard_normal(n + nb))
            st.y = torch.empty_like(st.x)
        else:
            st.mu, st.pts = _dev(_density(n, seed)), _dev(_star_points(case))
            st.out = torch.empty(st.pts.numel() // 2, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
    return st


def run(st):
    kind, case = st.kind, st.case
    if kind == "direct":
        s = kinterp.Solver(st.pr)
        mu, alpha = s.solve(st.pr.f)
        u = s.eval_targets(st.pr.targets, mu, alpha)
        s.close()
        return {"z": np.concatenate([mu, alpha]), "u": u}
    if kind == "refined":
        s = kinterp.Solver(st.pr, id_tol=case["id_tol"], mode=1)
        mu, alpha, _, _ = s.solve_refined(st.pr.f, rel_tol=REFINE_TOL)
        s.close()
        return {"z": np.concatenate([mu, alpha])}
    if kind == "integral":
        return kinterp.boundary_integral_solve(st.pr, st.pts, domain="disk", disk=(0.5, 0.5, 1.0))
    if kind == "batch":
        s = kinterp.BatchSolver(st.prs, id_tol=case["id_tol"], mode=1)
        mu, _, _ = s.solve_refined(st.f, rel_tol=REFINE_TOL)
        s.close()
        return mu
    if kind == "update":
        out = []
        for fr in st.frames:
            st.solver.update(fr)
            out.append(st.solver.solve(fr.f)[0])
        return out
    if kind == "adjoint":
        u = ki_autograd.target_potential(*st.leaves, st.targets, leaf_points=case["leaf"])
        J = ((u - st.u_star) ** 2).sum()
        return [u.detach(), *torch.autograd.grad(J, st.leaves)]
    if kind == "solve":
        st.solver.solve_device(st.f.data_ptr(), st.mu.data_ptr(),
                               st.alpha.data_ptr() if st.solver.n_border else None)
        return st.z
    if kind == "operator":
        st.solver.matvec_device(st.x.data_ptr(), st.y.data_ptr())
        return st.y
    st.solver.eval_domain_device(st.out.numel(), st.pts.data_ptr(), st.mu.data_ptr(), None,
                                 st.out.data_ptr(), domain="nodes")
    return st.out


# -------------------------------------------------------------------- work
def _factor_flops(nodes, sd, leaf):
    """Entries and pivoted QR steps of the boxes' compressions: every box has
    about leaf * sd columns and 2 (2 leaf + 128) sd rows of rank ~ 30 sd, and
    there are about 1.5 boxes for each leaf."""
    n, m, k = leaf * sd, 2 * (2 * leaf + 128) * sd, 30 * sd
    return 1.5 * nodes * sd / n * (20.0 * m * n + 4.0 * m * min(k, n) * n)


def work(case):
    """Inputs read and outputs written once; the compressions' arithmetic for
    a factorization, the pairs of an operator or a sum."""
    kind = case["kind"]
    sd = 2 if case.get("shape") == "stokes" else 1
    pair = 20.0 if sd == 2 else 13.0  # FP64 operations of a pair of nodes
    if kind == "batch":
        # mean of a log-uniform size
        a, b = case["nmin"], case["nmax"]
        nodes = case["count"] * (b - a) / max(math.log(b / a), 1e-9)
        pairs = case["count"] * (b * b - a * a) / max(2 * math.log(b / a), 1e-9)
        return {"bytes": 8.0 * 8 * nodes,
                "flops": _factor_flops(nodes, 1, case["leaf"]) + 2 * pair * pairs}
    n = case["n"] * (1.4 if kind == "integral" else 1.0)
    io = 8.0 * n * (6 + 2 * sd)
    if kind in ("direct", "refined"):
        fl = _factor_flops(n, sd, case["leaf"])
        return {"bytes": io, "flops": fl + (pair * n * n if kind == "refined" else 0.0)}
    if kind == "integral":
        nt = case["grid"] ** 2
        return {"bytes": io + 24.0 * nt, "flops": _factor_flops(n, 1, case["leaf"]) + 10.0 * nt * n}
    if kind == "update":
        # the boxes near the bump, twice, and two solves
        part = min(1.0, 6 * case["width"] / (2 * math.pi) + 0.1)
        return {"bytes": 2 * io, "flops": 2 * part * _factor_flops(n, 1, case["leaf"])}
    if kind == "adjoint":
        return {"bytes": 8.0 * n * 14,
                "flops": _factor_flops(n, 1, case["leaf"]) + 2 * 20.0 * n * (n + case["targets"])}
    if kind == "solve":
        # T, L, U and the inverse of a box's redundant block, read once
        return {"bytes": 8.0 * n * sd * (4 * 30 * sd + 2), "flops": 2.0 * n * sd * 4 * 30 * sd}
    if kind == "operator":
        return {"bytes": 8.0 * n * (6 + 2 * sd), "flops": pair * n * n}
    nt = case["grid"] ** 2
    return {"bytes": 8.0 * 7 * n + 24.0 * nt, "flops": 10.0 * nt * n}


# ------------------------------------------------------------------- exact
def _node_arrays(pr):
    p, q = _dev(pr.points).view(-1, 2), _dev(pr.normals).view(-1, 2)
    return p[:, 0], p[:, 1], q[:, 0], q[:, 1], _dev(pr.weights), _dev(pr.curvatures)


def _laplace_rows(tx, ty, g, diag=None):
    """Double-layer entries of the given target points; diag: the first
    target's node index, whose own entries take the curvature's limit."""
    x, y, nx, ny, w, k = g
    rx, ry = tx[:, None] - x[None, :], ty[:, None] - y[None, :]
    rho = rx * rx + ry * ry
    if diag is None:
        return -(w / (2 * math.pi)) * (rx * nx + ry * ny) / rho
    i = torch.arange(tx.numel(), device=tx.device)
    own = torch.zeros_like(rho, dtype=torch.bool)
    own[i, i + diag] = True
    a = -(w / (2 * math.pi)) * (rx * nx + ry * ny) / torch.where(own, torch.ones_like(rho), rho)
    return torch.where(own, (0.5 + k * w / (4 * math.pi)).expand_as(a), a)


def _stokes_rows(a, b, g):
    """Rows of the nodes a..b, both components each."""
    x, y, nx, ny, w, k = g
    n, m = x.numel(), b - a
    r = (x[a:b, None] - x[None, :], y[a:b, None] - y[None, :])
    rho = r[0] * r[0] + r[1] * r[1]
    i = torch.arange(m, device=x.device)
    rho[i, i + a] = 1.0
    pot = (w / math.pi) * (r[0] * nx + r[1] * ny) / (rho * rho)
    nn, tan = (nx, ny), (-ny, nx)
    out = torch.empty(m, 2, n, 2, dtype=torch.float64, device=x.device)
    for p in range(2):
        for q in range(2):
            e = pot * r[p] * r[q]
            e[i, i + a] = ((-0.5 if p == q else 0.0)
                           - k * w / (2 * math.pi) * tan[p] * tan[q])[a:b]
            out[:, p, :, q] = e + w * nn[p][a:b, None] * nn[q]
    return out.view(2 * m, 2 * n)


def _border(pr, tx, ty):
    """The holes' columns (logs; Stokeslets and rotlets) at the points."""
    cols = []
    for cx, cy, _, _ in np.asarray(pr.holes).reshape(-1, 4):
        rx, ry = tx - cx, ty - cy
        r2 = rx * rx + ry * ry
        if pr.pde == LAPLACE:
            cols.append(0.5 * torch.log(r2))
            continue
        s, lg = 1 / (4 * math.pi), -0.5 * torch.log(r2)
        for e in ((lg + rx * rx / r2, rx * ry / r2), (rx * ry / r2, lg + ry * ry / r2),
                  (ry / r2, -rx / r2)):
            cols.append(s * torch.stack(e, 1).reshape(-1))
    return torch.stack(cols, 1)


def _dense(pr):
    """The (bordered) system's matrix, made in blocks of rows."""
    g = _node_arrays(pr)
    x, y, w = g[0], g[1], g[4]
    sd = 2 if pr.pde == STOKES else 1
    n, holes = x.numel(), np.asarray(pr.holes).reshape(-1, 4)
    nb = (3 if sd == 2 else 1) * len(holes)
    A = torch.zeros(sd * n + nb, sd * n + nb, dtype=torch.float64, device="cuda")
    step = max(1, (1 << 25) // n)
    for a in range(0, n, step):
        b = min(n, a + step)
        A[sd * a:sd * b, :sd * n] = (_stokes_rows(a, b, g) if sd == 2 else
                                     _laplace_rows(x[a:b], y[a:b], g, a))
    if nb:
        A[:sd * n, sd * n:] = _border(pr, x, y)
        at = n - int(holes[:, 3].sum())
        for h, (_, _, _, cnt) in enumerate(holes):
            i = torch.arange(at, at + int(cnt), device="cuda")
            at += int(cnt)
            if sd == 1:
                A[n + h, i] = w[i]
                continue
            row = sd * n + 3 * h
            A[row, 2 * i], A[row + 1, 2 * i + 1] = w[i], w[i]
            A[row + 2, 2 * i], A[row + 2, 2 * i + 1] = w[i] * y[i], -w[i] * x[i]
        i = torch.arange(sd * n, sd * n + nb, device="cuda")
        A[i, i] = -1.0
    return A


def _gmres(A, b, steps=300):
    """Solution of A z = b by GMRES with two orthogonalizations a step; the
    rows are multiplied in blocks."""
    def mul(v):
        return torch.cat([r @ v for r in A.split(8192)])

    z = torch.zeros_like(b)
    for _ in range(2):  # the second solves for the first one's residual
        r = b - mul(z)
        beta = r.norm()
        V = torch.zeros(steps + 1, b.numel(), dtype=torch.float64, device="cuda")
        H = torch.zeros(steps + 1, steps, dtype=torch.float64, device="cuda")
        V[0] = r / beta
        for j in range(steps):
            u = mul(V[j])
            for _ in range(2):
                c = V[:j + 1] @ u
                u = u - c @ V[:j + 1]
                H[:j + 1, j] += c
            H[j + 1, j] = u.norm()
            V[j + 1] = u / H[j + 1, j]
            if j % 10 == 9:
                e = torch.zeros(j + 2, dtype=torch.float64, device="cuda")
                e[0] = beta
                c = torch.linalg.lstsq(H[:j + 2, :j + 1], e[:, None]).solution[:, 0]
                if (H[:j + 2, :j + 1] @ c - e).norm() < 1e-14 * b.norm():
                    break
        z = z + c @ V[:c.numel()]
    return z


def _solution(pr):
    """(mu, alpha) of the dense system."""
    A = _dense(pr)
    b = torch.zeros(A.shape[0], dtype=torch.float64, device="cuda")
    b[:pr.f.size] = _dev(pr.f)
    z = torch.linalg.solve(A, b) if A.shape[0] <= 20000 else _gmres(A, b)
    return z[:pr.f.size], z[pr.f.size:]


def _values(pr, pts, mu, alpha):
    """The solution at interior points, in blocks."""
    p, g = _dev(pts).view(-1, 2), _node_arrays(pr)
    out = []
    step = max(1, (1 << 25) // g[0].numel())
    for a in range(0, p.shape[0], step):
        tx, ty = p[a:a + step, 0], p[a:a + step, 1]
        if pr.pde == LAPLACE:
            u = _laplace_rows(tx, ty, g) @ mu
        else:
            rx, ry = tx[:, None] - g[0], ty[:, None] - g[1]
            rho = rx * rx + ry * ry
            s = (g[4] / math.pi) * (rx * g[2] + ry * g[3]) / (rho * rho) * (
                rx * mu[0::2] + ry * mu[1::2])
            u = torch.stack([(s * rx).sum(1), (s * ry).sum(1)], 1).reshape(-1)
        if alpha.numel():
            u = u + _border(pr, tx, ty) @ alpha
        out.append(u)
    return torch.cat(out)


def _in_star(pr, pts):
    """1 where a point is inside the node curve and not within 0.01 of a node."""
    p, x, y = _dev(pts).view(-1, 2), *_node_arrays(pr)[:2]
    yn = torch.roll(y, -1)
    out = []
    step = max(1, (1 << 25) // x.numel())
    for a in range(0, p.shape[0], step):
        tx, ty = p[a:a + step, 0, None], p[a:a + step, 1, None]
        near = (torch.sqrt((tx - x) ** 2 + (ty - y) ** 2) < 1e-2).any(1)
        right = x > tx
        cross = ((right & (y < ty) & (yn > ty)).sum(1) - (right & (y > ty) & (yn < ty)).sum(1))
        out.append(~near & (cross % 2 != 0))
    return torch.cat(out)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("direct", "refined"):
        pr = _problem(case, seed)
        mu, alpha = _solution(pr)
        out = {"z": torch.cat([mu, alpha]).cpu().numpy()}
        if kind == "direct":
            out["u"] = _values(pr, pr.targets, mu, alpha).cpu().numpy()
        return out
    if kind == "solve":
        return torch.cat(_solution(_problem(case, seed)))
    if kind == "batch":
        return torch.cat([_solution(p)[0] for p in _stars(case, seed)]).cpu().numpy()
    if kind == "update":
        return [_solution(fr)[0].cpu().numpy() for fr in _frames(case, seed)[1]]
    if kind == "integral":
        pr, pts = _annulus(case, seed), _annulus_points(case)
        u = _values(pr, pts, *_solution(pr))
        p = _dev(pts).view(-1, 2)
        bad = torch.sqrt((p[:, 0] - 0.5) ** 2 + (p[:, 1] - 0.5) ** 2) + 1e-2 > 1.0
        for cx, cy, rad, _ in pr.holes:
            bad |= torch.sqrt((p[:, 0] - cx) ** 2 + (p[:, 1] - cy) ** 2) - 1e-2 < rad
        return torch.where(bad, torch.zeros_like(u), u).cpu().numpy()
    if kind == "adjoint":
        pr, leaves = _adjoint_inputs(case, seed)
        for a in leaves:
            a.requires_grad_(True)
        pts, nrm, kap, w, f = leaves
        g = (pts[0::2], pts[1::2], nrm[0::2], nrm[1::2], w, kap)
        tg = _dev(pr.targets).view(-1, 2)
        mu = torch.linalg.solve(_laplace_rows(g[0], g[1], g, 0), f)
        u = _laplace_rows(tg[:, 0], tg[:, 1], g) @ mu
        J = ((u - _dev(pr.extra["u_star"])) ** 2).sum()
        return [u.detach(), *torch.autograd.grad(J, leaves)]
    if kind == "operator":
        pr = _problem(case, seed)
        A = _dense(pr)
        x = _dev(np.random.default_rng(seed).standard_normal(A.shape[0]))
        return torch.cat([r @ x for r in A.split(8192)])
    pr = G.star_case(n=case["n"], seed=seed, leaf_points=case["leaf"])
    pts = _star_points(case)
    u = _values(pr, pts, _dev(_density(case["n"], seed)), torch.zeros(0, device="cuda"))
    return torch.where(_in_star(pr, pts), u, torch.zeros_like(u))
