"""The FP64-accurate M2L on the tensor cores (ozaki_tc.cu) over every FMM order: parts of 48
operator rows (one at p <= 5, a second of one row at p = 6, three at p >= 9), one or two K chunks
(p <= 7 / p >= 8, with K steps left out at p = 8 and 9) and chunks of fewer than 128 rows, one and
several columns.

Reference: the plain FP64 operator on the same mesh.  The FP64-accurate operator is held to 1e-12
of it (2-norm): digits cut at 2^-48, the rest of the operator in float-float at about 2^-47 a term.
"""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", range(1, 11))
def test_orders(p, pibem_mod, synthetic):
    mesh, mask = synthetic.spheroid_mixed_case(15, seed=3)[:2]
    X = np.random.Generator(np.random.PCG64(p)).normal(size=(3, mesh.n_nodes))
    y = {}
    for mode in (pibem_mod.PRECISION_FP64, pibem_mod.PRECISION_FLOAT_FLOAT):
        g = pibem_mod.BEMSolver(fma_truncation_order=p, max_nodes_per_childless_block=10,
                                is_external_flow=1, precision_mode=mode)
        g.set_mesh(mesh.xyz, mesh.cells)
        g.set_bc(mask)
        y[mode] = g.system_matvec(X)
        alone = np.stack([g.system_matvec(X[r]) for r in range(3)])
        np.testing.assert_array_equal(alone, y[mode])
        g.close()
    assert rel(y[pibem_mod.PRECISION_FLOAT_FLOAT], y[pibem_mod.PRECISION_FP64]) < 1e-12
