"""The FP64 products of the factorisation on the tensor cores (kore_oz_selftest), entry by
entry against sums of exact products.

What the kernel may lose per real or imaginary part (csrc/gemm_oz.cu): 10.1 K 2^-60 of (largest
component of A's row) x (largest of B's column), A's columns and B's rows scaled against each
other, and one rounding per product, piece of the inner dimension and sum with C."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def product(lib, A1, B1, A2=None, B2=None, C=None, negate=0):
    from kore_gb300 import _lib as L
    S = A1.shape[0]
    # column-major: the transposes in C order
    ops = [None if m is None else np.ascontiguousarray(m.T, dtype=np.complex128) for m in (A1, B1, A2, B2)]
    out = np.array(np.full((S, S), np.nan) if C is None else C.T, dtype=np.complex128, order="C")
    rc = lib.kore_oz_selftest(0, S, *[L.ptr(m) if m is not None else None for m in ops], L.ptr(out), negate,
                              int(C is not None))
    assert rc == 0
    return out.T


def two_prod(a, b):
    """a b as p + e exactly (Dekker's product with Veltkamp's splitting)."""
    def split(x):
        c = 134217729.0 * x
        hi = c - (c - x)
        return hi, x - hi
    p = a * b
    ah, al = split(a)
    bh, bl = split(b)
    return p, ((ah * bh - p) + ah * bl + al * bh) + al * bl


def exact_part(terms, extra=0.0):
    """Correctly rounded extra + sum of the products a b of the (a, b) in terms."""
    s = [extra]
    for a, b in terms:
        p, e = two_prod(a, b)
        s += p.tolist() + e.tolist()
    return math.fsum(s)


def exact_entry(A, B, i, j):
    a, b = A[i], B[:, j]
    return complex(exact_part([(a.real, b.real), (-a.imag, b.imag)]), exact_part([(a.real, b.imag), (a.imag, b.real)]))


def entries(rng, S, n):
    edge = [0, S - 1, min(127, S - 1), min(128, S - 1), min(63, S - 1), min(64, S - 1)]
    return [(i, j) for i in edge[:2] for j in edge] + [tuple(rng.integers(S, size=2)) for _ in range(n)]


def comp_max(X, axis):
    return np.maximum(np.abs(X.real), np.abs(X.imag)).max(axis=axis)


def loss(A, B):
    return 10.1 * A.shape[1] * 2.0 ** -60 * np.outer(comp_max(A, 1), comp_max(B, 0))


@pytest.mark.parametrize("S", [224, 240, 292, 342, 448, 673, 1024])
def test_sums_are_exact(gpu_lib, S):
    """Entries whose digits are all 62 or 63, with signs that make both real products of the
    real part add: the largest sums there are (above 2^24 from 409 on for the pairs that weigh
    2^-40, were the inner dimension not cut)."""
    rng = np.random.default_rng(S)
    w = 2.0 ** (-6 - 7.0 * np.arange(7))
    part = lambda: rng.integers(62, 64, size=(S, S, 7)) @ w   # 49 bits: exact
    A, B = part() + 1j * part(), part() - 1j * part()
    C = product(gpu_lib, A, B)
    bound = loss(A, B)
    for i, j in entries(rng, S, 12):
        ref = exact_entry(A, B, i, j)
        # one rounding per piece of the last pass (two above 672) and one of their sum
        tol = 3 * 2.0 ** -53 * (np.abs(A[i]) @ np.abs(B[:, j])) * (1 if S > 672 else 0) + 2.0 ** -53 * abs(ref) + bound[i, j]
        assert abs(C[i, j].real - ref.real) <= tol and abs(C[i, j].imag - ref.imag) <= tol, (i, j, C[i, j], ref, tol)


@pytest.mark.parametrize("S", [1, 5, 16, 63, 64, 65, 129, 225, 449, 700, 1024])
@pytest.mark.parametrize("graded", [False, True])
def test_two_products(gpu_lib, S, graded):
    """C -= A1 B1 + A2 B2 at odd sizes, plain and graded by rows, columns and the inner index
    over sixteen orders of magnitude."""
    rng = np.random.default_rng(S + graded)

    def pair():
        A = rng.standard_normal((S, S)) + 1j * rng.standard_normal((S, S))
        B = rng.standard_normal((S, S)) + 1j * rng.standard_normal((S, S))
        return A, B
    (A1, B1), (A2, B2) = pair(), pair()
    lost = loss(A1, B1) + loss(A2, B2)
    if graded:
        g, h, u = (10.0 ** rng.uniform(-8, 8, S) for _ in range(3))
        A1, A2 = g[:, None] * A1 * u, g[:, None] * A2 / u
        B1, B2 = B1 / u[:, None] * h, B2 * u[:, None] * h
        lost = 4 * np.outer(g, h) * lost   # the inner scaling is a power of two from largest entries
    C0 = np.outer(comp_max(A1, 1), comp_max(B1, 0)) * rng.standard_normal((S, S))
    C = product(gpu_lib, A1, B1, A2, B2, C=C0, negate=1)
    for i, j in entries(rng, S, 12):
        r1, r2 = exact_entry(A1, B1, i, j), exact_entry(A2, B2, i, j)
        ref = C0[i, j] - r1 - r2
        mag = np.abs(A1[i]) @ np.abs(B1[:, j]) + np.abs(A2[i]) @ np.abs(B2[:, j]) + abs(C0[i, j])
        # at most two pieces of two products: four roundings of products, four of sums, and the
        # reference's two
        assert abs(C[i, j] - ref) <= 1.5 * (10 * 2.0 ** -53 * mag + lost[i, j]), (i, j, C[i, j], ref)


def test_zeros_infinities_subnormals(gpu_lib):
    """A zero row, column and inner index give zeros; rows and columns with an infinity or a NaN
    give NaN and touch nothing else; subnormal operands keep their bits."""
    S = 70
    rng = np.random.default_rng(0)
    A = rng.standard_normal((S, S)) + 1j * rng.standard_normal((S, S))
    B = rng.standard_normal((S, S)) + 1j * rng.standard_normal((S, S))
    A[3] = 0
    B[:, 5] = 0
    A[:, 7] = 0
    B[8] = 0
    ref = product(gpu_lib, A, B)
    assert np.all(ref[3] == 0) and np.all(ref[:, 5] == 0) and np.all(np.isfinite(ref))
    A2, B2 = A.copy(), B.copy()
    A2[10, 11] = np.inf
    B2[12, 13] = complex(0.0, np.nan)
    C = product(gpu_lib, A2, B2)
    bad = np.zeros((S, S), bool)
    bad[10] = bad[:, 13] = True
    assert np.all(np.isnan(C[bad].real)) and np.all(np.isnan(C[bad].imag)) and np.all(np.isfinite(C[~bad]))
    # subnormals: integers below 2^40 in units of 2^-1074 against integers, sums below 2^53
    T = rng.integers(-(1 << 20), 1 << 20, size=(S, S)) * 2.0 ** -1074 * (1 + 0j)
    N = rng.integers(-(1 << 10), 1 << 10, size=(S, S)) * (1.0 + 0j)
    exact = (np.rint(T.real * 2.0 ** 1000 * 2.0 ** 74) @ N.real) * 2.0 ** -1074
    np.testing.assert_array_equal(product(gpu_lib, T, N).real, exact)
    np.testing.assert_array_equal(product(gpu_lib, N, T).real, (N.real @ np.rint(T.real * 2.0 ** 1000 * 2.0 ** 74)) * 2.0 ** -1074)
