"""Workloads of the FMM-BEM library through its public Python entry points, for timing and for
comparing the results of two versions of the library.

    listed()             the standing workloads
    draw(rng)            one more of the same ranges
    prepare(case, seed)  mesh, handle and data a program has in hand before the call
    run(state)           the call, and what it returns
    work(case)           bytes and floating-point operations the call cannot do without
    exact(case, seed)    the same numbers from dense collocation matrices in 64 bits, without the
                         library (None where the dense form would take too long)

A case is a dict of plain values:
    kind   "solve"     pibem_solve_device: right-hand side, GMRES, phi and dphi/dn back
           "slots"     the same solves as a request stream through pibem_slots_*
           "fmm"       pibem_fmm_matvec (N phi and D dphi/dn), host arrays
           "system"    pibem_system_matvec and pibem_compute_rhs, host arrays
           "setup"     pibem_set_mesh + pibem_set_bc on an open handle, and the first rhs
           "gradient"  pibem_compute_normals + pibem_compute_gradients (after a solve)
    shape  "sphere" (interior, Dirichlet), "spheroid" / "blob" / "wigley" (exterior, mixed data),
           "cube" (sharp edges: double nodes and constraint lines)
    n      resolution: 6 n^2 + 2 nodes (cube: 6 (n + 1)^2; wigley: n cells along the hull)
    p, leaf, mode (0 FP64, 1 mixed, 2 float-float), prec (0 none, 1 leaf-block Jacobi, 2 ILU(0)),
    nrhs   columns

Solves are driven to a relative residual of 1e-12, where two correct solutions agree to about ten
digits whatever rounding the inner FP32 operator has; at a looser tolerance the iterates differ by
the condition number times that tolerance.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pi-bem_gb300"))
import pibem  # noqa: E402
import synthetic  # noqa: E402

TOLERANCE = 1e-12
QUAD, SINGULAR = 4, 5  # Gauss points per direction of a regular and of a singular cell
SLOTS = 6              # columns in flight of the request stream


def _case(name, kind, shape, n, p, leaf, mode, nrhs=1, prec=1):
    return dict(name=name, kind=kind, shape=shape, n=n, p=p, leaf=leaf, mode=mode, nrhs=nrhs, prec=prec)


def listed():
    return [
        # One small Dirichlet problem, a few milliseconds of dependent small kernels: latency.
        _case("solve sphere 1538", "solve", "sphere", 16, 4, 30, 1),
        # The benchmark's default workload: one mixed solve at 98,306 nodes.
        _case("solve spheroid 98306", "solve", "spheroid", 128, 8, 40, 1),
        # A thin ship hull at the highest order (121 coefficients per expansion), 55,250 nodes.
        _case("solve wigley 55250", "solve", "wigley", 288, 10, 40, 1),
        # Many load cases on one mesh (the batched workload): 16 columns share each application.
        _case("solve blob 23816 x16", "solve", "blob", 63, 8, 40, 1, nrhs=16),
        # The plain FP64 path, for users who want no mixed precision.
        _case("solve fp64 spheroid 13826", "solve", "spheroid", 48, 8, 40, 0),
        # The reference's own preconditioner, ILU(0) of the near field.
        _case("solve ilu spheroid 2402", "solve", "spheroid", 20, 6, 20, 0, prec=2),
        # A CAD-like body with sharp edges: constraint lines, whose right-hand side needs the L2
        # projections of normals and surface gradients.
        _case("solve cube 3750", "solve", "cube", 24, 6, 20, 1, nrhs=2),
        # A server's view: twelve right-hand sides that arrive while others are being solved.
        _case("slots blob 6146", "slots", "blob", 32, 6, 30, 1, nrhs=12),
        # The smallest call: one FMM product at the reference's default order and leaf size.
        _case("fmm 386", "fmm", "sphere", 8, 6, 20, 0),
        # One FP64-accurate operator application and right-hand side on a large hull.
        _case("system wigley 198109", "system", "wigley", 546, 10, 40, 2),
        # A new mesh: octree, lists, near-field integrals, tables, boundary flags.
        _case("setup blob 23816", "setup", "blob", 63, 8, 40, 1),
        # Velocities on the surface after a solve: the L2 projections of three load cases.
        _case("gradient spheroid 41336", "gradient", "spheroid", 83, 4, 40, 0, nrhs=3),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "solve", "slots", "fmm", "system", "setup", "gradient"])
    shape = rng.choice(["sphere", "spheroid", "blob", "wigley", "cube"])
    mode = rng.choice([1, 1, 1, 2, 0])
    p, leaf, prec, nrhs = rng.choice([4, 5, 6, 7, 8, 10]), rng.choice([20, 30, 40]), 1, 1
    if kind == "solve":
        if mode == 1:
            n = _log(rng, 8, 100)
            nrhs = rng.choice([1, 1, 2, 3, 5, 16]) if n <= 40 else 1
        else:
            n = _log(rng, 8, 40)
            if n <= 16 and rng.random() < 0.5:
                prec = 2
            if mode == 0:
                p = min(p, 8)
    elif kind == "slots":
        mode, n, nrhs = 1, _log(rng, 10, 36), rng.choice([3, 5, 8, 12])
    elif kind in ("fmm", "system"):
        n, nrhs = _log(rng, 6, 110), rng.choice([1, 1, 2, 4])
        if kind == "fmm":
            mode, p, nrhs = 0, min(p, 8), min(nrhs, 2)
    elif kind == "setup":
        n = _log(rng, 8, 80)
    else:
        mode, n, nrhs = 0, _log(rng, 8, 100), rng.choice([1, 2, 3, 5])
    if shape == "wigley":
        n = max(24, int(4.2 * n))
    return {k: v for k, v in _case("", kind, shape, n, p, leaf, mode, nrhs, prec).items() if k != "name"}


def _mesh(case, seed):
    """Mesh, Dirichlet mask, double-node CSR (or None, None), exterior problem or not."""
    n, shape = case["n"], case["shape"]
    if shape == "sphere":
        mesh = synthetic.cube_sphere(n)
        return mesh, np.ones(mesh.n_nodes, np.uint8), None, None, 0
    if shape == "cube":
        mesh, off, ids, face = synthetic.sharp_cube(n)
        mask = np.zeros(mesh.n_nodes, np.uint8)
        mask[np.unique(mesh.cells[np.isin(face, (0, 4))])] = 1
        return mesh, mask, off, ids, 1
    if shape == "spheroid":
        mesh = synthetic.spheroid(n)
        return mesh, synthetic.mixed_bc_by_cell_centroid(mesh), None, None, 1
    if shape == "blob":
        mesh = synthetic.perturbed_sphere(n, seed)
        return mesh, synthetic.random_plane_mask(mesh, seed), None, None, 1
    mesh = synthetic.wigley_hull(n, max(3, n // 4), max(2, n // 6))
    return mesh, synthetic.mixed_bc_by_cell_centroid(mesh, z_split=-0.5 * 0.0625), None, None, 1


def _data(case, mesh, mask, seed):
    """Boundary data of nrhs point-source fields: tmp_rhs, phi and dphi/dn, (nrhs, N) each."""
    out = [], [], []
    for r in range(case["nrhs"]):
        rng = np.random.Generator(np.random.PCG64([int(seed), r]))
        q = rng.uniform(-1.0, 1.0, 8)
        if case["shape"] == "wigley":
            src = synthetic.sources_in_wigley(rng, 8)
        else:
            src = synthetic.sources_in_ball(rng, 8)
            if case["shape"] == "sphere":  # interior problem: the sources outside
                src *= (1.6 + np.linalg.norm(src, axis=1))[:, None] / np.linalg.norm(src, axis=1)[:, None]
        for v, o in zip(synthetic.point_source_data(mesh, mask, src, q), out):
            o.append(v)
    return tuple(np.stack(o) for o in out)


def prepare(case, seed):
    mesh, mask, off, ids, exterior = _mesh(case, seed)
    tmp, phi, dphi = _data(case, mesh, mask, seed)
    solver = pibem.BEMSolver(
        fma_truncation_order=case["p"], num_octree_levels=10, max_nodes_per_childless_block=case["leaf"],
        quadrature_order=QUAD, singular_quadrature_order=SINGULAR, is_external_flow=exterior,
        precision_mode=case["mode"], preconditioner=case["prec"], solver_tolerance=TOLERANCE,
        solver_max_steps=2000, gmres_restart=100)
    s = dict(case=case, solver=solver, mesh=mesh, mask=mask, off=off, ids=ids, tmp=tmp, phi=phi, dphi=dphi)
    kind = case["kind"]
    if kind != "setup":
        solver.set_mesh(mesh.xyz, mesh.cells, off, ids)
        if kind != "fmm":
            solver.set_bc(mask)
    if kind == "solve":
        known = torch.as_tensor(mask == 1, device="cuda")
        s["d_tmp"] = torch.as_tensor(tmp, device="cuda")
        zero = torch.zeros_like(s["d_tmp"])
        s["d_phi"] = torch.where(known, s["d_tmp"], zero)
        s["d_dphi"] = torch.where(known, zero, s["d_tmp"])
        torch.cuda.synchronize()
    return s


def _run_slots(s):
    """Half of the slots are taken at once; a waiting request joins between two steps."""
    solver, tmp = s["solver"], s["tmp"]
    phi, dphi = np.empty_like(tmp), np.empty_like(tmp)
    solver.slots_open(SLOTS)
    waiting, left, room = list(range(len(tmp))), len(tmp), SLOTS // 2
    while left:
        while waiting and room and solver.slots_submit(waiting[0], tmp[waiting[0]]) is not None:
            waiting.pop(0)
            room -= 1
        solver.slots_step(16 if waiting else 0)
        room = SLOTS if not waiting else 1
        while (got := solver.slots_collect()) is not None:
            phi[got[0]], dphi[got[0]] = got[1], got[2]
            left -= 1
    solver.slots_close()
    return {"phi": phi, "dphi": dphi}


def run(state):
    s, solver = state, state["solver"]
    kind = s["case"]["kind"]
    if kind == "solve":
        solver.solve_device(s["case"]["nrhs"], s["d_phi"].data_ptr(), s["d_dphi"].data_ptr(), s["d_tmp"].data_ptr())
        return {"phi": s["d_phi"], "dphi": s["d_dphi"]}
    if kind == "slots":
        return _run_slots(s)
    if kind == "fmm":
        return solver.fmm_matvec(s["phi"], s["dphi"])
    if kind == "system":
        return solver.system_matvec(s["tmp"]), solver.rhs(s["tmp"])
    if kind == "setup":
        solver.set_mesh(s["mesh"].xyz, s["mesh"].cells, s["off"], s["ids"])
        solver.set_bc(s["mask"])
        return {"alpha": solver.alpha(), "rhs": solver.rhs(s["tmp"])}
    return {"normals": solver.normals(), "gradients": solver.gradients(s["phi"], s["dphi"])}


def _nodes(case):
    """Nodes of the mesh (wigley: before the sides and the lid share theirs, below 1 % more)."""
    n = case["n"]
    if case["shape"] == "cube":
        return 6 * (n + 1) ** 2
    if case["shape"] == "wigley":
        return 2 * n * max(3, n // 4) + n * max(2, n // 6)
    return 6 * n * n + 2


def work(case):
    N, R, K, leaf = _nodes(case), case["nrhs"], (case["p"] + 1) ** 2, case["leaf"]
    # Of a surface mesh, per node: about 15 leaf near-field entries, 110 / leaf M2L pairs, and
    # three rows of K expansion values (P2M, L2P).  One application reads the near field and
    # the rows once for all columns.
    near, pairs, rows = 15 * leaf * N, 110 * N / leaf, 3 * N * K
    flops = R * (2 * near + 2 * K * K * pairs + 2 * rows)
    vectors = 8 * N * R
    kind = case["kind"]
    if kind in ("solve", "slots"):
        steps = 20 * N ** 0.15 * (0.5 if case["prec"] == 2 else 1.0)
        size = 4 if case["mode"] == 1 else 8
        return {"bytes": steps * (size * (near + rows) + 2 * vectors), "flops": steps * (flops + 4 * N * R * min(steps, 100))}
    if kind == "fmm":
        return {"bytes": 8 * 2 * (near + rows) + 4 * vectors, "flops": 2 * flops}
    if kind == "system":
        return {"bytes": 2 * (8 * (near + rows) + 2 * vectors), "flops": 2 * flops}
    if kind == "setup":
        # both layers of every near-field entry from about 4 cells of 16 points, written once
        return {"bytes": 2 * 8 * near, "flops": near * 4 * QUAD ** 2 * 12.0 + 2 * flops}
    # mass matrix products of about 40 CG steps, 3 components a column, 9 entries a row
    return {"bytes": 40 * 3 * 8 * N * (R + 1) * 3, "flops": 40 * 3 * N * (R + 1) * 2 * 9}


# ---- the dense form in 64 bits ---------------------------------------------------------------


def _gauss(n):
    x, w = np.polynomial.legendre.leggauss(n)
    return 0.5 * (x + 1.0), 0.5 * w


def _telles(n, end):
    """The cubic transformation of a Gauss rule on [0, 1] with its points drawn to one end."""
    x, w = _gauss(n)
    g, b = 2.0 * x - 1.0, 2.0 * end - 1.0
    return 0.5 * (((g - b) ** 3 + 4.0 * b) / 4.0 + 1.0), w * 0.75 * (g - b) ** 2


def _rule(xi, wi, eta, we):
    return np.repeat(eta, len(xi)), np.tile(xi, len(eta)), np.outer(we, wi).ravel()


def _shape(eta, xi):
    return np.stack([(1 - xi) * (1 - eta), xi * (1 - eta), (1 - xi) * eta, xi * eta], axis=1)


def _points(v, eta, xi, w):
    """Points, unit normals, weights and tangents of bilinear cells v (C, 4, 3) at one rule."""
    dev = v.device
    t = lambda a: torch.as_tensor(a, device=dev)  # noqa: E731
    dxi, deta = t(np.stack([-(1 - eta), 1 - eta, -eta, eta], 1)), t(np.stack([-(1 - xi), -xi, 1 - xi, xi], 1))
    x = torch.einsum("qa,cak->cqk", t(_shape(eta, xi)), v)
    tx, ty = torch.einsum("qa,cak->cqk", dxi, v), torch.einsum("qa,cak->cqk", deta, v)
    c = torch.linalg.cross(tx, ty)
    J = c.norm(dim=2)
    return x, c / J[..., None], J * t(w)[None, :], (tx, ty, dxi, deta)


def _layers(x, xq, nq, wq):
    """Double- and single-layer kernels times weights; x (M, 3) against points of each row."""
    d = xq - x
    r2 = (d * d).sum(-1)
    inv = torch.rsqrt(r2) / (4.0 * math.pi)
    single = inv * wq
    return -(d * nq).sum(-1) / r2 * single, single


def _dense(mesh, off, ids, phi, dphi, matrices=False):
    """N phi and D dphi/dn (columns (N, R)) by direct collocation, or the matrices N and D."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    xyz, cells = torch.as_tensor(mesh.xyz, device=dev), torch.as_tensor(mesh.cells.astype(np.int64), device=dev)
    N, C = xyz.shape[0], cells.shape[0]
    v = xyz[cells]
    g, gw = _gauss(QUAD)
    eta, xi, w = _rule(g, gw, g, gw)
    sh = torch.as_tensor(_shape(eta, xi), device=dev)
    xq, nq, wq, _ = _points(v, eta, xi, w)
    xq, nq, wq = xq.reshape(-1, 3), nq.reshape(-1, 3), wq.reshape(-1)
    if matrices:
        A, B = (torch.zeros(N, N, dtype=torch.float64, device=dev) for _ in range(2))
    else:
        fq = torch.einsum("qa,car->cqr", sh, phi[cells]).reshape(C * len(w), -1)
        gq = torch.einsum("qa,car->cqr", sh, dphi[cells]).reshape(C * len(w), -1)
        A, B = torch.zeros_like(phi), torch.zeros_like(dphi)
    # (node, cell, vertex at the node): cells that touch a node or one of its doubles
    sets = np.arange(N) if off is None else np.asarray(ids)
    owner = np.arange(N) if off is None else np.repeat(np.arange(N), np.diff(off))
    flat = mesh.cells.astype(np.int64).ravel()
    order = np.argsort(flat, kind="stable")
    start = np.searchsorted(flat[order], np.arange(N + 1))
    cnt = start[sets + 1] - start[sets]
    at = np.repeat(start[sets] - np.concatenate([[0], np.cumsum(cnt)[:-1]]), cnt) + np.arange(cnt.sum())
    inc = np.stack([np.repeat(owner, cnt), order[at] // 4, order[at] % 4], 1)
    # of a cell that meets the node twice (a collapsed edge) the first vertex counts
    inc = inc[np.lexsort((inc[:, 2], inc[:, 1], inc[:, 0]))]
    keep = np.ones(len(inc), bool)
    keep[1:] = (inc[1:, 0] != inc[:-1, 0]) | (inc[1:, 1] != inc[:-1, 1])
    inc = torch.as_tensor(inc[keep], device=dev)
    rows = max(1, int(6e7) // (C * len(w)))
    for a in range(0, N, rows):
        b = min(N, a + rows)
        kn, kd = _layers(xyz[a:b, None, :], xq[None], nq[None], wq[None])
        mine = inc[(inc[:, 0] >= a) & (inc[:, 0] < b)]
        for k in (kn, kd):  # the cells at the node come from the singular rule below
            k.view(b - a, C, -1)[mine[:, 0] - a, mine[:, 1]] = 0.0
        if matrices:
            for k, M in ((kn, A), (kd, B)):
                M[a:b].index_add_(1, cells.ravel(), torch.einsum("mcq,qa->mca", k.view(b - a, C, -1), sh).reshape(b - a, -1))
        else:
            A[a:b], B[a:b] = kn @ fq, kd @ gq
    for j in range(4):
        sub = inc[inc[:, 2] == j]
        tx, tw = _telles(SINGULAR, j & 1)
        ty, tv = _telles(SINGULAR, j >> 1)
        eta, xi, w = _rule(tx, tw, ty, tv)
        x, n, wt, _ = _points(v[sub[:, 1]], eta, xi, w)
        kn, kd = _layers(xyz[sub[:, 0], None, :], x, n, wt)
        sh4 = torch.as_tensor(_shape(eta, xi), device=dev)
        for k, M, f in ((kn, A, phi), (kd, B, dphi)):
            val = k @ sh4  # (incidences, 4)
            if matrices:
                M.index_put_((sub[:, :1].expand(-1, 4), cells[sub[:, 1]]), val, accumulate=True)
            else:
                M.index_add_(0, sub[:, 0], torch.einsum("ia,iar->ir", val, f[cells[sub[:, 1]]]))
    return A, B


def _projected(mesh, phi, dphi):
    """Q1 projections of the normal and of grad phi + n dphi/dn: CG on the mass matrix."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    xyz, cells = torch.as_tensor(mesh.xyz, device=dev), torch.as_tensor(mesh.cells.astype(np.int64), device=dev)
    g, gw = _gauss(QUAD)
    eta, xi, w = _rule(g, gw, g, gw)
    sh = torch.as_tensor(_shape(eta, xi), device=dev)
    _, n, wq, (tx, ty, dxi, deta) = _points(xyz[cells], eta, xi, w)
    a11, a12, a22 = (tx * tx).sum(2), (tx * ty).sum(2), (ty * ty).sum(2)
    det = a11 * a22 - a12 * a12
    fields = [n]
    for f, d in zip(phi, dphi):
        fx, fe = torch.einsum("qa,ca->cq", dxi, f[cells]), torch.einsum("qa,ca->cq", deta, f[cells])
        cx, ce = (a22 * fx - a12 * fe) / det, (a11 * fe - a12 * fx) / det
        fields.append(cx[..., None] * tx + ce[..., None] * ty + torch.einsum("qa,ca->cq", sh, d[cells])[..., None] * n)
    F = torch.cat(fields, 2)
    b = torch.zeros(xyz.shape[0], F.shape[2], dtype=torch.float64, device=dev)
    b.index_add_(0, cells.ravel(), torch.einsum("qa,cqk,cq->cak", sh, F, wq).reshape(-1, F.shape[2]))
    Mc = torch.einsum("qa,qb,cq->cab", sh, sh, wq)
    M = torch.sparse_coo_tensor(torch.stack([cells.repeat_interleave(4, 1).ravel(), cells.repeat(1, 4).ravel()]),
                                Mc.ravel(), (xyz.shape[0],) * 2).coalesce()
    diag = torch.zeros(xyz.shape[0], dtype=torch.float64, device=dev)
    diag.index_add_(0, cells.ravel(), torch.diagonal(Mc, dim1=1, dim2=2).reshape(-1))
    x, r = torch.zeros_like(b), b.clone()
    z = r / diag[:, None]
    d, rz = z.clone(), (r * z).sum(0)
    for _ in range(400):
        q = M @ d
        alpha = rz / (d * q).sum(0)
        x, r = x + alpha * d, r - alpha * q
        if float((r.norm(dim=0) / b.norm(dim=0)).max()) < 1e-15:
            break
        z = r / diag[:, None]
        new = (r * z).sum(0)
        d, rz = z + new / rz * d, new
    return x[:, :3].contiguous(), x[:, 3:].reshape(-1, len(phi), 3).permute(1, 0, 2).contiguous()


def exact(case, seed):
    kind = case["kind"]
    N = _nodes(case)
    solves = kind in ("solve", "slots")
    if case["shape"] == "cube" and (solves or kind == "setup"):
        return None  # the constraint lines of sharp edges have no plain dense form here
    if kind != "gradient" and N > (9000 if solves else 32000):
        return None  # longer than some seconds
    mesh, mask, off, ids, exterior = _mesh(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    tmp, phi, dphi = (torch.as_tensor(v, device=dev) for v in _data(case, mesh, mask, seed))
    if kind == "gradient":
        n, g = _projected(mesh, phi, dphi)
        return {"normals": n, "gradients": g}
    if kind == "fmm":
        a, b = _dense(mesh, off, ids, phi.T.contiguous(), dphi.T.contiguous())
        return a.T.contiguous(), b.T.contiguous()
    dir_ = torch.as_tensor(mask == 1, device=dev)[None]
    one, zero = torch.ones_like(tmp[:1]), torch.zeros_like(tmp)
    if solves:
        A, B = _dense(mesh, off, ids, None, None, matrices=True)
        alpha = -A.sum(1) - exterior
        A.diagonal().add_(alpha)
        known = torch.where(dir_, tmp, zero).T
        flux = torch.where(dir_, zero, tmp).T
        rhs = -A @ known + B @ flux
        x = torch.linalg.solve(torch.where(dir_, -B, A), rhs).T
        return {"phi": torch.where(dir_, tmp, x), "dphi": torch.where(dir_, x, tmp)}
    # columns: N on the Dirichlet part, on the Neumann part and on 1; D the other way round
    f = torch.cat([torch.where(dir_, tmp, zero), torch.where(dir_, zero, tmp), one]).T.contiguous()
    a, b = (v.T for v in _dense(mesh, off, ids, f, f))
    R = case["nrhs"]
    alpha = -a[2 * R] - exterior
    rhs = -(a[:R] + alpha * torch.where(dir_, tmp, zero)) + b[R:2 * R]
    if kind == "setup":
        return {"alpha": alpha, "rhs": rhs}
    return a[R:2 * R] - b[:R] + alpha * torch.where(dir_, zero, tmp), rhs
