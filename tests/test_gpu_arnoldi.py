"""The Arnoldi step (krylov.cu arnoldi_*_kernel) where its loops change shape: meshes smaller than
a block's chunk of rows, restarts below and above the 64 basis vectors a sweep of the dots takes,
several columns (four at a time in the preconditioner) and the preconditioner variants.

Oracle: the CPU oracle's GMRES solve of the same FMM system.  Both are driven to a relative
residual of 1e-12; with condition numbers below 1e4 the solutions agree to 1e-8.
"""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu

CASES = [
    # n, restart, preconditioner, mode, columns
    (2, 100, 1, 1, 1),
    (2, 100, 0, 0, 3),
    (5, 10, 1, 1, 5),
    (8, 12, 1, 0, 2),
    (8, 80, 0, 1, 1),
    (8, 120, 2, 0, 2),
    (11, 70, 0, 0, 4),
    (23, 64, 1, 1, 6),
]


@pytest.mark.parametrize("n,restart,prec,mode,nrhs", CASES)
def test_arnoldi_shapes(n, restart, prec, mode, nrhs, pibem_mod, oracle_mod, synthetic):
    mesh, mask = synthetic.spheroid_mixed_case(n, seed=1)[:2]
    tmp = np.stack([synthetic.spheroid_mixed_case(n, seed=1 + r, mesh=mesh)[2] for r in range(nrhs)])
    g = pibem_mod.BEMSolver(fma_truncation_order=5, max_nodes_per_childless_block=20,
                            is_external_flow=1, precision_mode=mode, preconditioner=prec,
                            gmres_restart=restart, solver_tolerance=1e-12, solver_max_steps=6000)
    g.set_mesh(mesh.xyz, mesh.cells)
    g.set_bc(mask)
    phi, dphi, st = g.solve(tmp)
    assert st["relative_residual"] <= 1e-12
    o = oracle_mod.Oracle(p=5, levels=10, max_nodes=20, external=True)
    o.set_mesh(mesh.xyz, mesh.cells)
    o.set_bc(mask)
    for r in range(nrhs):
        ophi, odphi, _, _ = o.solve(tmp[r], tol=1e-12, max_steps=6000)
        assert rel(phi[r], ophi) < 1e-8
        assert rel(dphi[r], odphi) < 1e-8
    # a column alone has the same bits
    p1, d1, _ = g.solve(tmp[nrhs - 1])
    np.testing.assert_array_equal(p1, phi[nrhs - 1])
    np.testing.assert_array_equal(d1, dphi[nrhs - 1])
    g.close()
