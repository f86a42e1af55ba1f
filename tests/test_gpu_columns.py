"""The operator's kernels that take several columns at a time (near field, P2M, M2P, L2P and the
translations) at column counts that fill, miss and exceed their groups of 2 and 4, and at FMM
orders with one to four coefficients per lane (K = 9, 36, 81, 121) and leaves of few nodes.

A column has the same bits alone and in a batch, in each arithmetic.  The FP64 products are held to
1e-10 of the oracle (2-norm), the bound of the parity tests."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [2, 5, 8, 10])
def test_column_counts(p, pibem_mod, oracle_mod, synthetic, monkeypatch):
    mesh, mask = synthetic.spheroid_mixed_case(11, seed=4)[:2]
    n = mesh.n_nodes
    X = np.random.Generator(np.random.PCG64(p)).normal(size=(6, n))
    o = oracle_mod.Oracle(p=p, levels=10, max_nodes=7, external=True)
    o.set_mesh(mesh.xyz, mesh.cells)
    o.set_bc(mask)
    monkeypatch.setenv("PIBEM_MATVEC_FP32", "1")  # the mixed handle's product: its FP32 operator
    for mode in (pibem_mod.PRECISION_FP64, pibem_mod.PRECISION_FLOAT_FLOAT, pibem_mod.PRECISION_MIXED):
        g = pibem_mod.BEMSolver(fma_truncation_order=p, max_nodes_per_childless_block=7,
                                is_external_flow=1, precision_mode=mode)
        g.set_mesh(mesh.xyz, mesh.cells)
        g.set_bc(mask)
        alone = np.stack([g.system_matvec(x) for x in X])
        for R in (2, 3, 5, 6):
            np.testing.assert_array_equal(g.system_matvec(X[:R]), alone[:R])
        N1, D1 = zip(*(g.fmm_matvec(X[r], X[5 - r]) for r in range(3)))
        N2, D2 = g.fmm_matvec(X[:2], X[5:3:-1])
        N3, D3 = g.fmm_matvec(X[:3], X[5:2:-1])
        np.testing.assert_array_equal(N2, N1[:2])
        np.testing.assert_array_equal(D2, D1[:2])
        np.testing.assert_array_equal(N3, N1)
        np.testing.assert_array_equal(D3, D1)
        if mode == pibem_mod.PRECISION_FP64:
            oN, oD = o.fmm_matvec(X[0], X[5])
            assert rel(N3[0], oN) < 1e-10 and rel(D3[0], oD) < 1e-10
        g.close()


@pytest.mark.parametrize("leaf,leaves", [(40, (200, 1216)), (12, (1217, 2432)), (4, (2433, 9000))])
def test_warps_per_leaf(leaf, leaves, pibem_mod, oracle_mod, synthetic, monkeypatch):
    """P2M and L2P with four, two and one warps per leaf (by the number of leaves): FP64 products
    against the oracle (1e-10), the FP32 operator against the FP64 one (2e-5, the bound of the level
    passes' tests) and a column alone against the batch (bitwise)."""
    mesh, mask = synthetic.spheroid_mixed_case(40, seed=6)[:2]
    X = np.random.Generator(np.random.PCG64(leaf)).normal(size=(5, mesh.n_nodes))
    o = oracle_mod.Oracle(p=4, levels=10, max_nodes=leaf, external=True)
    o.set_mesh(mesh.xyz, mesh.cells)
    o.set_bc(mask)
    monkeypatch.setenv("PIBEM_MATVEC_FP32", "1")
    y = {}
    for mode in (pibem_mod.PRECISION_FP64, pibem_mod.PRECISION_MIXED):
        g = pibem_mod.BEMSolver(fma_truncation_order=4, max_nodes_per_childless_block=leaf,
                                is_external_flow=1, precision_mode=mode)
        g.set_mesh(mesh.xyz, mesh.cells)
        g.set_bc(mask)
        assert leaves[0] <= g.tree_info()["n_leaves"] <= leaves[1]
        y[mode] = g.system_matvec(X)
        np.testing.assert_array_equal(np.stack([g.system_matvec(x) for x in X]), y[mode])
        if mode == pibem_mod.PRECISION_FP64:
            N, D = g.fmm_matvec(X[0], X[1])
        g.close()
    oN, oD = o.fmm_matvec(X[0], X[1])
    assert rel(N, oN) < 1e-10 and rel(D, oD) < 1e-10
    for r in range(5):
        assert rel(y[pibem_mod.PRECISION_MIXED][r], y[pibem_mod.PRECISION_FP64][r]) < 2e-5
