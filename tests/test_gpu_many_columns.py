"""The calls with host arrays at column counts beyond what one launch's grid takes (65,535 blocks a
dimension): every column has the bits it has alone.  And a call that fails leaves nothing behind for
the next one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

R = 70000  # the product of N and D runs 2 R columns


@pytest.mark.parametrize("leaf", [3, 30])
@pytest.mark.parametrize("mode", ["PRECISION_FP64", "PRECISION_MIXED", "PRECISION_FLOAT_FLOAT"])
def test_many_columns(mode, leaf, pibem_mod, synthetic, monkeypatch):
    mesh = synthetic.spheroid(3)
    n = mesh.n_nodes
    some = [0, 4095, 4096, 8191, 65535, 65536, R - 1]
    X = np.random.Generator(np.random.PCG64(leaf)).normal(size=(R, n))
    g = pibem_mod.BEMSolver(fma_truncation_order=1, max_nodes_per_childless_block=leaf, is_external_flow=1,
                            precision_mode=getattr(pibem_mod, mode))
    g.set_mesh(mesh.xyz, mesh.cells)
    g.set_bc(synthetic.mixed_bc_by_cell_centroid(mesh))
    calls = {"fmm": lambda x: np.stack(g.fmm_matvec(x, x[:, ::-1]), 1), "system": g.system_matvec, "rhs": g.rhs,
             "preconditioner": g.apply_preconditioner, "gradients": lambda x: g.gradients(x, x)}
    for name, f in calls.items():
        Y = f(X)
        for r in some:
            np.testing.assert_array_equal(np.asarray(f(X[r:r + 1]))[0], Y[r], err_msg=f"{name} {r}")
    g.close()


def test_failed_call_leaves_no_error(pibem_mod, synthetic):
    mesh = synthetic.spheroid(3)
    with pytest.raises(pibem_mod.PibemError):
        pibem_mod.BEMSolver(device=99)
    g = pibem_mod.BEMSolver(fma_truncation_order=2)
    g.set_mesh(mesh.xyz, mesh.cells)
    g.close()
