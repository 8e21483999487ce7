"""A shift's results do not depend on how many shifts share the plan: factors, solves and
eigenpairs are bit for bit those of the shift alone, in both precisions and in every compiled
sweep variant."""
import numpy as np
import pytest
import scipy.sparse as ss

pytestmark = pytest.mark.gpu


def blocks(sizes, seed):
    """A block-tridiagonal pencil with dense diagonal blocks and sparse couplings."""
    from kore_gb300 import Layout, Pencil
    rng = np.random.default_rng(seed)
    K = len(sizes)
    rows = [[None] * K for _ in range(K)]
    for i, s in enumerate(sizes):
        rows[i][i] = ss.csr_matrix(rng.standard_normal((s, s)) + 1j * rng.standard_normal((s, s)) + 4 * s * np.eye(s))
        for j in (i - 1, i + 1):
            if 0 <= j < K:
                rows[i][j] = ss.random(s, sizes[j], density=min(1.0, 6.0 / sizes[j]), random_state=rng, format="csr") * 1j
    A = ss.bmat(rows, format="csr").astype(complex)
    n = A.shape[0]
    lay = Layout(n=n, N1=max(sizes), nb=K, perm=np.arange(n), block_sizes=np.array(sizes, dtype=np.int32),
                 block_ell=np.arange(K), sections=("u",), coupling=1)
    return Pencil(A, ss.diags(rng.uniform(0.5, 1.0, n), format="csr"), layout=lay)


def same_as_alone(p, sig, precision, seed):
    rng = np.random.default_rng(seed)
    b = rng.standard_normal((p.n, len(sig))) + 1j * rng.standard_normal((p.n, len(sig)))
    p.factor_shifts(sig, precision)
    x = p.solve(b)
    for s in sorted({0, len(sig) // 2, len(sig) - 1}):
        p.factor(sig[s], precision)
        np.testing.assert_array_equal(p.solve(b[:, s]), x[:, s])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("sizes,nshift", [([24] * 20, 8), ([48] * 40, 4), ([96] * 12, 16), ([100, 97] * 6, 5), ([132] * 9, 24),
                                          ([200] * 8, 6), ([360, 240] * 2, 3)])
def test_solves(gpu_lib, sizes, nshift, precision):
    with blocks(sizes, len(sizes)) as p:
        same_as_alone(p, 1j * np.linspace(-1.0, 1.0, nshift), precision, nshift)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_sweep_variants(gpu_lib, precision):
    """All sweep variants give the same bits."""
    from kore_gb300.solver import sweep_variant
    rng = np.random.default_rng(0)
    with blocks([100, 97] * 8, 3) as p:
        p.factor(0.3j, precision)
        b = rng.standard_normal(p.n) + 1j * rng.standard_normal(p.n)
        ref = p.solve(b)
        try:
            for cps in (2, 3, 4):
                for chunk in (8192, 16384):
                    sweep_variant(cps, chunk)
                    np.testing.assert_array_equal(p.solve(b), ref)
        finally:
            sweep_variant(0, 0)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_eigenpairs(gpu_lib, case, precision):
    """Targets together and through fewer slots (single re-factorised slots) as each alone."""
    from kore_gb300 import Pencil, eigs_targets, layout_from_params
    meta, A, B = case("shell_m1_ek1e-4")
    targets, seeds = [1.0j, 0.6j, 0.05 + 1.4j, 0.8j], [3, 4, 5, 6]
    with Pencil(A, B, layout=layout_from_params(meta)) as p:
        kw = dict(which="TM", precision=precision, tol=1e-13, maxit=100)
        alone = [eigs_targets(p, [t], 6, seeds=[s], **kw)[0] for t, s in zip(targets, seeds)]
        for slots in (4, 2):
            for (lam, X, _), (lam1, X1, _) in zip(eigs_targets(p, targets, 6, seeds=seeds, slots=slots, **kw), alone):
                np.testing.assert_array_equal(lam, lam1)
                np.testing.assert_array_equal(X, X1)
