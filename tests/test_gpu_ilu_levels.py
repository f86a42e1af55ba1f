"""ILU(0) substitutions by the shape of the triangles' levels (krylov.cu): meshes numbered at random,
whose levels are few and wide, run a launch per level; meshes numbered along the surface, whose levels
hold a few rows, run one block per column, with the solution in shared memory up to 25,600 nodes (200 KB)
and in global memory beyond.  All against the oracle's preconditioner at the bound of the other ILU
tests, 1e-10 relative, two columns at once; and the two forms against each other, bit for bit."""
import ctypes as C

import numpy as np
import pytest

import kernel_harness as kh
from conftest import rel

pytestmark = pytest.mark.gpu


def renumbered(synthetic, mesh, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    new = rng.permutation(mesh.n_nodes)
    old = np.argsort(new)
    return synthetic.Mesh(mesh.xyz[old], new[mesh.cells].astype(mesh.cells.dtype), mesh.normals[old])


def solver(pibem_mod, mesh, mask, leaf, **kw):
    g = pibem_mod.BEMSolver(fma_truncation_order=2, max_nodes_per_childless_block=leaf, is_external_flow=1,
                            precision_mode=pibem_mod.PRECISION_FP64, **kw)
    g.set_mesh(mesh.xyz, mesh.cells)
    g.set_bc(mask)
    return g


# (resolution, random numbering, most launches of an application or None: a launch per level)
@pytest.mark.parametrize("n,shuffled,launches", [(65, False, 4), (66, False, 4), (48, True, None), (66, True, None)])
def test_apply(n, shuffled, launches, pibem_mod, oracle_mod, synthetic):
    mesh = synthetic.spheroid(n)
    if shuffled:
        mesh = renumbered(synthetic, mesh, 1)
    mask = synthetic.mixed_bc_by_cell_centroid(mesh)
    o = oracle_mod.Oracle(p=2, levels=10, max_nodes=4, external=True)
    o.set_mesh(mesh.xyz, mesh.cells)
    o.set_bc(mask)
    apply, _ = o.preconditioner(2)
    g = solver(pibem_mod, mesh, mask, 4, preconditioner=2)
    V = np.random.Generator(np.random.PCG64(n)).normal(size=(2, mesh.n_nodes))
    l0 = pibem_mod.launch_count()
    Z = g.apply_preconditioner(V)
    count = pibem_mod.launch_count() - l0
    assert count <= launches if launches else count > 100
    for r in range(2):
        assert rel(Z[r], apply(V[r])) < 1e-10
    g.close()


def test_solve_with_wide_levels(pibem_mod, synthetic):
    """The level launches inside the GMRES cycle graph: the same bits step by step (profiling on),
    and the solution of the leaf-block Jacobi solve to 1e-8 at a tolerance of 1e-11."""
    mesh = renumbered(synthetic, synthetic.spheroid(48), 2)
    mask = synthetic.mixed_bc_by_cell_centroid(mesh)
    src = synthetic.sources_in_ball(np.random.Generator(np.random.PCG64(3)), 4)
    tmp = synthetic.point_source_data(mesh, mask, src, np.array([1.0, -0.5, 0.7, 0.2]))[0]
    out = {}
    for prec in (1, 2):
        g = solver(pibem_mod, mesh, mask, 4, preconditioner=prec, solver_tolerance=1e-11)
        phi, dphi, _ = g.solve(tmp)
        out[prec] = np.concatenate([phi, dphi])
        if prec == 2:
            g.set_profiling(1)
            phi1, dphi1, _ = g.solve(tmp)
            np.testing.assert_array_equal(phi1, phi)
            np.testing.assert_array_equal(dphi1, dphi)
        g.close()
    assert rel(out[2], out[1]) < 1e-8


@pytest.mark.parametrize("n", [3, 700, 25600, 25601])
def test_both_forms_round_alike(n):
    """Random factors, rows of 1 to 600 entries (more than the 512 that a warp loads at once), pivots
    without short reciprocals: the two forms' sums and quotients are the same."""
    lib = kh.load()
    rng = np.random.Generator(np.random.PCG64(n))
    cols = []
    for i in range(n):
        k = int(rng.choice([0, 3, 9, 40])) if n > 1000 else int(rng.choice([0, 3, 40, 600]))
        cols.append(np.unique(np.append(rng.integers(0, n, k), i)))
    ptr = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int64)
    col = np.concatenate(cols).astype(np.int32)
    diag = np.array([ptr[i] + np.searchsorted(cols[i], i) for i in range(n)], np.int64)
    val = rng.normal(size=len(col)) / 40.0
    val[diag] = rng.uniform(0.5, 2.0, n)

    def by_level(lower):
        lev = np.zeros(n, int)
        for i in range(n) if lower else range(n - 1, -1, -1):
            c = cols[i][cols[i] < i] if lower else cols[i][cols[i] > i]
            if len(c):
                lev[i] = lev[c].max() + 1
        count = np.bincount(lev)
        return np.concatenate([[0], np.cumsum(count)]).astype(np.int64), np.argsort(lev, kind="stable").astype(np.int32)

    lo, up = by_level(True), by_level(False)
    z0 = rng.normal(size=(2, n))
    z = {}
    for levels in (0, 1):
        z[levels] = z0.copy()
        assert lib.kh_ilu(n, 2, kh.ptr(ptr, C.c_int64), kh.ptr(col, C.c_int32), kh.ptr(val, C.c_double),
                          kh.ptr(diag, C.c_int64), len(lo[0]) - 1, kh.ptr(lo[0], C.c_int64), kh.ptr(lo[1], C.c_int32),
                          len(up[0]) - 1, kh.ptr(up[0], C.c_int64), kh.ptr(up[1], C.c_int32), levels,
                          kh.ptr(z[levels], C.c_double)) == 0
    np.testing.assert_array_equal(z[0], z[1])


def test_wait_that_gives_up_has_its_own_code():
    """Row 0 of the forward order waits for a row that its own warp only takes later (16 warps): the
    bounded wait runs out, the kernel returns and the error flag is the substitutions' own."""
    lib = kh.load()
    n = 40
    ptr = np.arange(n + 1, dtype=np.int64)
    ptr[18:] += 1  # row 17 = [16, 17], the others their diagonal
    col = np.insert(np.arange(n), 17, 16).astype(np.int32)
    diag = np.array([ptr[i] + (i == 17) for i in range(n)], np.int64)
    val = np.ones(n + 1)
    rows = np.arange(n, dtype=np.int32)
    rows[[0, 17]] = rows[[17, 0]]  # row 17 first, row 16 at place 16: both of warp 0
    lptr = np.array([0, n], np.int64)
    z = np.ones((1, n))
    assert lib.kh_ilu(n, 1, kh.ptr(ptr, C.c_int64), kh.ptr(col, C.c_int32), kh.ptr(val, C.c_double),
                      kh.ptr(diag, C.c_int64), 1, kh.ptr(lptr, C.c_int64), kh.ptr(rows, C.c_int32),
                      1, kh.ptr(lptr, C.c_int64), kh.ptr(np.arange(n, dtype=np.int32), C.c_int32), 0,
                      kh.ptr(z, C.c_double)) == 2
