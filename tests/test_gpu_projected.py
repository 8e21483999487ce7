"""Projected eigenproblems of every size class the Krylov-Schur kernel takes (a basis of two
vectors up to the 64 its shared memory holds, odd sizes, more and fewer entries than
threads), through whole eigensolves against the oracle's eigenvalues."""
import numpy as np
import pytest

from oracle.eps_ref import eig_residuals, shift_invert_eigs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which", ["TM", "TI"])
@pytest.mark.parametrize("nev,ncv", [(1, 2), (1, 3), (2, 7), (4, 16), (5, 31), (5, 33), (8, 47), (10, 63), (10, 64)])
def test_basis_sizes(gpu_lib, case, nev, ncv, which):
    from kore_gb300 import EPS, Pencil, layout_from_params
    meta, A, B = case("shell_m1_ek1e-4")
    tau = complex(*meta["tau"])
    with Pencil(A, B, layout=layout_from_params(meta)) as p:
        E = EPS()
        E.setOperators(p)
        E.setProblemType(EPS.ProblemType.GNHEP)
        E.setDimensions(nev, ncv)
        E.setTolerances(1e-13, 2000)
        E.setWhichEigenpairs(which)
        E.setTarget(tau)
        E.setFromOptions({"kore_precision": "fp64", "kore_seed": 3})
        E.solve()
    lam, X = E.eigenvalues(), E.eigenvectors()
    assert len(lam) >= nev, E.stats
    # genuine eigenpairs; the eigenvalues nearest the target also agree with the oracle's to
    # the bar of the eigenvalue comparison
    assert eig_residuals(A, B, lam[:nev], X[:, :nev]).max() < 1e-12
    if which == "TM" and ncv >= 7:
        ref, _ = shift_invert_eigs(A, B, tau, nev, "TM")
        assert max(np.min(np.abs(lam - r)) / abs(r) for r in ref[:nev]) < 1e-11
