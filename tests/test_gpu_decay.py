"""FP64 forced solves whose solution falls off over many orders of magnitude with the degree:
each degree's block carries the relative accuracy that the same block cyclic reduction has in
NumPy's FP64, down to blocks of 1e-20 of the largest (products that are accurate only relative
to the largest entries of rows and columns lose the small blocks)."""
import numpy as np
import pytest
import scipy.sparse as ss

pytestmark = pytest.mark.gpu


def reduction(band):
    """Factors of the block cyclic reduction of K blocks (band[k]: L, D, U of block row k)."""
    K = len(band)
    D, L, U = ({k: band[k][i] for k in range(K)} for i in (1, 0, 2))
    act, levels = list(range(K)), []
    while len(act) > 1:
        odd, even = act[1::2], act[0::2]
        right = {b: act[i + 1] if i + 1 < len(act) else None for i, b in enumerate(act)}
        left = {b: act[i - 1] if i else None for i, b in enumerate(act)}
        inv = {j: np.linalg.inv(D[j]) for j in odd}
        G = {j: inv[j] @ L[j] for j in odd}
        H = {j: inv[j] @ U[j] for j in odd if right[j] is not None}
        levels.append((odd, even, left, right, inv, G, H, dict(L), dict(U)))
        for b in even:
            l, r, lo, up = left[b], right[b], L[b], U[b]
            if l is not None:
                D[b] = D[b] - lo @ H[l]
                L[b] = -lo @ G[l]
            if r is not None:
                D[b] = D[b] - up @ G[r]
                U[b] = -up @ H[r] if r in H else None
        act = even
    return levels, np.linalg.inv(D[act[0]])


def solve(factors, f):
    levels, top = factors
    f, z, x = [v.copy() for v in f], {}, {}
    for odd, even, left, right, inv, G, H, L, U in levels:
        for j in odd:
            z[j] = inv[j] @ f[j]
        for b in even:
            if left[b] is not None:
                f[b] = f[b] - L[b] @ z[left[b]]
            if right[b] is not None:
                f[b] = f[b] - U[b] @ z[right[b]]
    x[0] = top @ f[0]
    for odd, even, left, right, inv, G, H, L, U in reversed(levels):
        for j in odd:
            x[j] = z[j] - G[j] @ x[left[j]]
            if right[j] is not None:
                x[j] = x[j] - H[j] @ x[right[j]]
    return np.stack([x[k] for k in range(len(f))])


def residual_long(M, b, x):
    """b - M x in long double."""
    re, im = M.data.real.astype(np.longdouble), M.data.imag.astype(np.longdouble)
    xr, xi = x.real[M.indices], x.imag[M.indices]
    return b - (np.add.reduceat(re * xr - im * xi, M.indptr[:-1]) + 1j * np.add.reduceat(re * xi + im * xr, M.indptr[:-1]))


@pytest.mark.parametrize("omega", [0.3, 1.1, -1.7])
def test_small_blocks_keep_their_accuracy(gpu_lib, omega):
    from kore_gb300 import Pencil
    from kore_gb300.assembly import forcing_vector, hydro_params, hydro_pencil
    from kore_gb300.structure import layout_from_params
    m, N, lmax, Ek, ricb = 1, 48, 100, 1e-4, 0.35
    A, B, norm = hydro_pencil(m, 1, Ek, N, lmax, ricb, with_norm=True)
    lay = layout_from_params(hydro_params(m, 1, Ek, N, lmax, ricb))
    b = forcing_vector(m, 1, N, lmax, ricb, 10).toarray().ravel() / norm
    with Pencil(A, B, layout=lay) as p:
        p.factor(1j * omega, "fp64")
        x = p.solve(b)
    # the same rows and unknowns by degree, rows scaled by powers of two
    K = len(lay.block_sizes)
    M = (A - 1j * omega * B).tocsr()[lay.perm][:, lay.perm].tocsr()
    scale = 2.0 ** -np.floor(np.log2(np.abs(M).max(axis=1).toarray().ravel()))
    M, f = (ss.diags(scale) @ M).tocsr(), scale * b[lay.perm]
    row = lambda k, q: M[k * N:(k + 1) * N, q * N:(q + 1) * N].toarray() if 0 <= q < K else np.zeros((N, N))
    factors = reduction([[row(k, k + d) for d in (-1, 0, 1)] for k in range(K)])
    plain = solve(factors, f.reshape(K, N)).ravel()
    true = plain.astype(np.clongdouble)
    for _ in range(8):
        true = true + solve(factors, residual_long(M, f, true).astype(complex).reshape(K, N)).ravel()
    size = np.linalg.norm(true.astype(complex).reshape(K, N), axis=1)
    err = lambda y: np.linalg.norm((y - true).astype(complex).reshape(K, N), axis=1) / size
    e, e0 = err(x[lay.perm]), err(plain)
    # two roundings of one algorithm: the errors differ by chance, sixteenfold at most allowed
    # against the largest of the eleven blocks around
    near = np.array([e0[max(0, k - 5):k + 6].max() for k in range(K)])
    keep = size > 1e-20 * size.max()
    assert keep.sum() > K // 2 and size[keep].min() < 1e-15 * size.max()
    assert np.all(e[keep] <= 16 * near[keep]), [(k, size[k], e[k], near[k]) for k in np.flatnonzero(keep & (e > 16 * near))]
