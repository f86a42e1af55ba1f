"""P2M tables (setup.cu) formed run of leaves by run of leaves: the same bits whether the work buffer
holds all points' expansions, a few leaves' or less than one leaf's, and the monopole sums against
numpy to 1e-13 (2-norm; some hundred FP64 terms a value)."""
import ctypes as C

import numpy as np
import pytest

import kernel_harness as kh
from test_gpu_m2l_error import basis

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [1, 8, 10])
def test_runs_of_leaves(p):
    lib = kh.load()
    rng = np.random.Generator(np.random.PCG64(p))
    K = (p + 1) ** 2
    K4 = (K + 3) // 4 * 4
    points = [5, 1, 33, 64, 200, 2, 31]  # per leaf; four vertices a point among the leaf's rows
    Q = sum(points)
    order = rng.permutation(Q)  # the leaves' points are not contiguous
    row_ptr, contrib_ptr, contrib_q, leaf_of = [0], [0], [], np.empty(Q, int)
    for leaf, n in enumerate(points):
        mine = np.sort(order[sum(points[:leaf]):sum(points[:leaf]) + n])
        leaf_of[mine] = leaf
        rows = 4 + leaf
        row_of = {(q, j): r for q in mine for j, r in enumerate(rng.permutation(rows)[:4])}
        used = 0
        for r in range(rows):
            mine_r = sorted(int(q) * 4 + j for (q, j), v in row_of.items() if v == r)
            if mine_r:
                contrib_q += mine_r
                contrib_ptr.append(len(contrib_q))
                used += 1
        row_ptr.append(row_ptr[-1] + used)
    row_ptr, contrib_ptr = np.array(row_ptr, np.int64), np.array(contrib_ptr, np.int64)
    contrib_q = np.array(contrib_q, np.int32)
    L = len(points)
    center, delta = rng.normal(size=(L, 3)), rng.uniform(0.5, 2.0, L)
    rel_pos = rng.uniform(-0.5, 0.5, (Q, 3))
    qpts = np.ascontiguousarray(center[leaf_of] + delta[leaf_of, None] * rel_pos)
    qnrm = rng.normal(size=(Q, 3))
    qw = rng.normal(size=(Q, 4))
    point_bytes = 2 * K4 * 8
    out = []
    for work in (1 << 30, 70 * point_bytes, 1):
        T = np.zeros((2, row_ptr[-1], K4))
        assert lib.kh_p2m_tables(p, L, kh.ptr(row_ptr, C.c_int64), kh.ptr(contrib_ptr, C.c_int64),
                                 kh.ptr(contrib_q, C.c_int32), kh.ptr(center, C.c_double), kh.ptr(delta, C.c_double),
                                 Q, kh.ptr(qpts, C.c_double), kh.ptr(qnrm, C.c_double), kh.ptr(qw, C.c_double),
                                 C.c_int64(work), kh.ptr(T[0], C.c_double), kh.ptr(T[1], C.c_double)) == 0
        out.append(T)
    np.testing.assert_array_equal(out[1], out[0])
    np.testing.assert_array_equal(out[2], out[0])
    rel = (qpts - center[leaf_of]) / delta[leaf_of, None]
    unit = basis(p, rel)
    want = np.stack([qw.ravel()[contrib_q[a:b]] @ unit[contrib_q[a:b] >> 2]
                     for a, b in zip(contrib_ptr[:-1], contrib_ptr[1:])])
    assert np.linalg.norm(out[0][1][:, :K] - want) <= 1e-13 * np.linalg.norm(want)
    assert np.isfinite(out[0]).all() and (out[0][:, :, K:] == 0).all()
