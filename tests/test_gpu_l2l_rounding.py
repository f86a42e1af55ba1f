"""L2L of the FP32 operator (levels.cu) against the same sums on the host, bit for bit: one chain of
fused multiply-adds in ascending order up to K = 81, four chains of a quarter each, added pairwise,
beyond (p = 9, 10), whose rounding a longer chain would double.  Boxes of all, of one and of no
octant per block, one column and three."""
import ctypes as C

import numpy as np
import pytest

import kernel_harness as kh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [1, 3])
@pytest.mark.parametrize("p", [3, 8, 9, 10])
def test_same_sums_as_the_host(p, R):
    lib = kh.load()
    rng = np.random.Generator(np.random.PCG64(p))
    K, parents = (p + 1) ** 2, 40
    counts = [70, 1, 0, 33, 400, 0, 17, 64]
    oct_ = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    n = int(oct_[-1])
    box = (parents + rng.permutation(n)).astype(np.int32)
    par = rng.integers(0, parents, n).astype(np.int32)
    L0 = rng.normal(size=(parents + n, R, K)).astype(np.float32)
    got, want = L0.copy(), L0.copy()
    for ref, L in ((0, got), (1, want)):
        assert lib.kh_l2l(p, R, parents + n, n, kh.ptr(box, C.c_int32), kh.ptr(par, C.c_int32),
                          kh.ptr(oct_, C.c_int32), ref, kh.ptr(L, C.c_float)) == 0
    np.testing.assert_array_equal(got, want)
