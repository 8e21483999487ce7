"""Factorisation at block sizes around the edges of its panels, tiles and register
layouts (32 and 16 columns per panel, 128 rows and 8 or 32 columns per update tile, 256,
512 and 1024 rows per panel CTA), against the oracle's sparse LU.

Blocks are random with a dominant, cyclically shifted diagonal, so that every pivot lies
off the diagonal; couplings are sparse, as the pencils' are.  The normwise backward error
of elimination with partial pivoting on these blocks (no growth) is at most a few S u per
block of the chain: 4 S K u is allowed in FP64; mixed solves are refined to 1e-15."""
import numpy as np
import pytest
import scipy.sparse as ss

from oracle.eps_ref import forced_solve, solve_residual

pytestmark = pytest.mark.gpu


def pencil(sizes, seed):
    from kore_gb300 import Layout, Pencil
    rng = np.random.default_rng(seed)
    K = len(sizes)
    rows = []
    for i, s in enumerate(sizes):
        D = rng.standard_normal((s, s)) + 1j * rng.standard_normal((s, s))
        D += 4 * s * np.roll(np.eye(s), s // 3 + 1, axis=0)
        row = [None] * K
        row[i] = ss.csr_matrix(D)
        for j in (i - 1, i + 1):
            if 0 <= j < K:
                row[j] = ss.random(s, sizes[j], density=min(1.0, 6.0 / sizes[j]), random_state=rng, format="csr") * 1j
        rows.append(row)
    A = ss.bmat(rows, format="csr").astype(complex)
    n = A.shape[0]
    B = ss.diags(rng.uniform(0.5, 1.0, n), format="csr")
    lay = Layout(n=n, N1=max(sizes), nb=K, perm=np.arange(n), block_sizes=np.array(sizes, dtype=np.int32),
                 block_ell=np.arange(K), sections=("u",), coupling=1)
    return A, B, Pencil(A, B, layout=lay)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("sizes,nshift", [
    ([3, 1, 4], 1), ([31, 33, 32], 1), ([48, 24, 48, 24, 48], 3), ([65] * 4, 1), ([129, 127, 128], 1),
    ([132] * 9, 24), ([256, 255], 1), ([257, 260], 1), ([512, 480], 1), ([513, 516], 1), ([700, 350, 700], 1),
    ([1000, 1024], 1)])
def test_block_shapes(gpu_lib, sizes, nshift, precision):
    A, B, p = pencil(sizes, sum(sizes) + nshift)
    rng = np.random.default_rng(3)
    n = A.shape[0]
    sig = 1j * np.linspace(-1.0, 1.0, nshift) if nshift > 1 else np.array([0.3j])
    b = rng.standard_normal((n, nshift)) + 1j * rng.standard_normal((n, nshift))
    with p:
        p.factor_shifts(sig, precision)
        x = p.solve(b, refine_tol=1e-15)
    tol = 4 * max(sizes) * len(sizes) * 1.1e-16 if precision == "fp64" else 1e-14
    for s in {0, nshift // 2, nshift - 1}:
        M = (A - sig[s] * B).tocsr()
        assert solve_residual(M, x[:, s], b[:, s]) <= tol, s
        xr = forced_solve(M, b[:, s])
        assert np.linalg.norm(x[:, s] - xr) <= 1e-10 * np.linalg.norm(xr), s


@pytest.mark.parametrize("S", [1, 5, 16, 33, 67, 127, 128, 129, 144, 256, 260, 513, 1024])
def test_tc_gemm_tile_edges(gpu_lib, S):
    """The complex64 tensor-core product around its 128 x 128 x 32 tile and at odd sizes
    (columns off the 16-byte boundary).  3xTF32 with FP32 accumulation relative to
    sum |a||b|: the dropped lo lo product and the rounding of lo (2^-21 each) and the
    accumulation of S terms and twelve products, sqrt(12 S) 2^-24."""
    import ctypes
    err = ctypes.c_double(-1.0)
    assert gpu_lib.kore_tc_selftest(0, S, 6, ctypes.byref(err)) == 0
    assert 0.0 <= err.value < 2 * 2.0 ** -21 + (12 * S) ** 0.5 * 2.0 ** -24, err.value


@pytest.mark.parametrize("nshift,k", [(1, 1), (1, 3), (3, 9), (9, 9)])
def test_columns_equal_vectors(gpu_lib, nshift, k):
    """Right-hand sides side by side (kore_solve_cols, one vector for all included) give bit
    for bit what the same vectors give one after another (kore_solve)."""
    import ctypes
    from kore_gb300 import _lib as L
    A, B, p = pencil([33, 31, 32, 40], 5)
    rng = np.random.default_rng(1)
    n = A.shape[0]
    b = rng.standard_normal((n, k)) + 1j * rng.standard_normal((n, k))
    with p:
        p.factor_shifts(1j * np.linspace(0.1, 1.0, nshift), "mixed")
        rows, ref = np.ascontiguousarray(b.T), np.empty((k, n), dtype=complex)
        assert p.lib.kore_solve(p._plan, L.ptr(rows), L.ptr(ref), k, 0.0, ctypes.byref(L.Stats())) == 0
        np.testing.assert_array_equal(p.solve(b), ref.T)
        np.testing.assert_array_equal(p.solve(np.asfortranarray(b)), ref.T)
        one = np.broadcast_to(b[:, :1], (n, k))
        np.testing.assert_array_equal(p.solve(one), p.solve(np.array(one)))
        bad = b.copy()
        bad[n // 2, k - 1] = np.inf
        with pytest.raises(L.KoreError) as e:
            p.solve(bad)
        assert e.value.status == 8   # KORE_ENAN
