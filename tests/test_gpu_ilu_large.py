"""ILU(0) substitutions of a mesh whose solution values do not fit a block's shared memory
(n beyond 228 KB / 8 bytes), where they are handed on through global memory: two columns against
the oracle's preconditioner at the bound of the smaller meshes' tests, 1e-10 relative."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


def test_apply_beyond_shared_memory(pibem_mod, oracle_mod, synthetic):
    mesh, mask = synthetic.spheroid_mixed_case(71, seed=2)[:2]
    assert mesh.n_nodes * 8 > 228 * 1024
    o = oracle_mod.Oracle(p=2, levels=10, max_nodes=4, external=True)
    o.set_mesh(mesh.xyz, mesh.cells)
    o.set_bc(mask)
    apply, _ = o.preconditioner(2)
    g = pibem_mod.BEMSolver(fma_truncation_order=2, max_nodes_per_childless_block=4, is_external_flow=1,
                            precision_mode=pibem_mod.PRECISION_FP64, preconditioner=2)
    g.set_mesh(mesh.xyz, mesh.cells)
    g.set_bc(mask)
    V = np.random.Generator(np.random.PCG64(5)).normal(size=(2, mesh.n_nodes))
    Z = g.apply_preconditioner(V)
    for r in range(2):
        assert rel(Z[r], apply(V[r])) < 1e-10
    g.close()
