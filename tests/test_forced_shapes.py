"""forced_sweep refuses right-hand sides whose length is not the pencil's, in a single group of
frequencies as in several (host logic on a stand-in pencil that reshapes as Pencil.solve does)."""
import numpy as np
import pytest

from kore_gb300.solver import forced_sweep


class StandIn:
    n = 4

    def factor_shifts(self, sigmas, precision):
        pass

    def solve(self, rhs, refine_tol=0.0, stats=False):
        x = np.ascontiguousarray(np.asarray(rhs, dtype=complex).reshape(self.n, -1))
        return (x, {"solve_resid_max": 0.0}) if stats else x


@pytest.mark.parametrize("F,group", [(1, 16), (2, 16), (4, 2)])
@pytest.mark.parametrize("columns", [False, True])
def test_wrong_length_is_refused(F, group, columns):
    b = np.ones((8, F)) if columns else np.ones(8)
    with pytest.raises(ValueError):
        forced_sweep(StandIn(), np.linspace(0, 1, F), b, "fp64", group=group)


@pytest.mark.parametrize("F,group", [(1, 16), (3, 16), (5, 2), (0, 16)])
def test_right_length(F, group):
    X, times = forced_sweep(StandIn(), np.linspace(0, 1, F), np.arange(4.0), "fp64", group=group, scale=2.0)
    np.testing.assert_array_equal(X, np.repeat(np.arange(4.0)[:, None], F, axis=1) / 2)
    assert X.dtype == complex and len(times) == -(-F // group)
