"""Error of the FP64-accurate M2L at the orders that run seven digits (p = 9, 10; ozaki_tc.cu): by
degree of the output coefficient, since the low degrees hide the high ones in any norm over all of
them.  The kernel's error is relative to the largest entries of the expansion and of the operator
row, the float-float GEMM's to each term; the digits have to be no less exact at any degree,
whatever the sources: smooth or random strengths on planes through the box, sources in its corners
(expansions that fall slowly with the degree), sources at its centre (expansions that fall fast).

Bound: the float-float GEMM's own 2-norm error against sums in long double on the same pairs.  With
exact group sums the digits' error is below a third of it at every degree."""
import ctypes as C

import numpy as np
import pytest

import kernel_harness as kh

pytestmark = pytest.mark.gpu
SOURCES, POINTS = 48, 200


def basis(p, r):
    """(len(r), K) scaled real multipole terms of unit sources at r: rho^n P~_n^m (cos, -sin) m beta."""
    rho = np.linalg.norm(r, axis=1)
    x, beta = r[:, 2] / rho, np.arctan2(r[:, 1], r[:, 0])
    s = np.sqrt(np.maximum(0.0, 1.0 - x * x))
    P = np.zeros((p + 1, p + 1, len(r)))
    for m in range(p + 1):
        P[m, m] = 1.0 if m == 0 else -np.sqrt((2 * m - 1) / (2 * m)) * s * P[m - 1, m - 1]
        for n in range(m + 1, p + 1):
            a = (2 * n - 1) * x * P[n - 1, m]
            b = np.sqrt((n - 1) ** 2 - m * m) * P[n - 2, m] if n > m + 1 else 0.0
            P[n, m] = (a - b) / np.sqrt(n * n - m * m)
    out = np.empty((len(r), (p + 1) ** 2))
    for n in range(p + 1):
        out[:, n * n] = rho**n * P[n, 0]
        for m in range(1, n + 1):
            out[:, n * n + 2 * m - 1] = rho**n * P[n, m] * np.cos(m * beta)
            out[:, n * n + 2 * m] = -(rho**n) * P[n, m] * np.sin(m * beta)
    return out


def expansions(p, kind, rng):
    E = np.empty((SOURCES, (p + 1) ** 2))
    for i in range(SOURCES):
        r = rng.uniform(-0.5, 0.5, (POINTS, 3))
        if kind == "plane":
            nv = rng.normal(size=3)
            nv /= np.linalg.norm(nv)
            r -= np.outer(r @ nv - rng.uniform(-0.3, 0.3), nv)
            r = np.clip(r, -0.5, 0.5)
        elif kind == "corners":
            r = np.where(r < 0, -0.5, 0.5) * (1.0 - 0.02 * np.abs(r))
        else:
            r *= 0.1
        w = rng.normal(size=POINTS) if i % 2 else 1.0 + 0.3 * r @ rng.normal(size=3)
        E[i] = w @ basis(p, r) / POINTS
    return E


@pytest.mark.parametrize("kind", ["plane", "corners", "centre"])
@pytest.mark.parametrize("p", [9, 10])
def test_no_less_exact_than_float_float(p, kind):
    lib = kh.load()
    rng = np.random.Generator(np.random.PCG64(p))
    K = (p + 1) ** 2
    g = np.arange(-3, 4, dtype=np.int32)
    off = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    off = np.ascontiguousarray(off[np.abs(off).max(1) >= 2])
    off = np.ascontiguousarray(off[rng.permutation(len(off))[:60]])
    nof = len(off)
    E = expansions(p, kind, rng)
    pairs = np.empty(E.shape + (2,), np.float32)
    pairs[..., 0] = E
    pairs[..., 1] = E - pairs[..., 0]
    # chunks of 128 and 28 pairs, of 48 and of 1
    op = np.repeat(np.arange(nof, dtype=np.int32), [156 if o == 0 else 48 if o < 50 else 1 for o in range(nof)])
    src = rng.integers(0, SOURCES, len(op)).astype(np.int32)
    T = np.empty((nof + 16, K, K))
    lib.kh_ops(p, nof, kh.ptr(off, C.c_int32), kh.ptr(T, C.c_double))
    El = pairs.astype(np.longdouble).sum(-1)
    exact = np.empty((len(op), K), np.longdouble)
    for o in range(nof):
        q = op == o
        exact[q] = El[src[q]] @ T[o].astype(np.longdouble)
    degree = np.sqrt(np.arange(K) + 0.5).astype(int)
    err = {}
    for digits in (0, 1):
        Y = np.zeros((len(op), K, 2), np.float32)
        assert lib.kh_m2l(p, nof, kh.ptr(off, C.c_int32), SOURCES, kh.ptr(pairs, C.c_float), len(op),
                          kh.ptr(src, C.c_int32), kh.ptr(op, C.c_int32), digits, kh.ptr(Y, C.c_float)) == 0
        d = Y.astype(np.longdouble).sum(-1) - exact
        err[digits] = np.array([float(np.linalg.norm(d[:, degree == n].astype(float)) /
                                      np.linalg.norm(exact[:, degree == n].astype(float))) for n in range(p + 1)])
    print(p, kind, "float-float", err[0], "digits", err[1])
    assert (err[1] <= err[0]).all()
