"""Status of a solve from the device error flag and its NaN state: a wait that ran out is reported
as such also when the entries it left unset made the residual a NaN (no GPU)."""
import pytest


@pytest.mark.parametrize("flag,nan,status", [(0, 0, 0), (0, 1, 8), (2, 0, 4), (2, 1, 4), (3, 0, 6), (3, 1, 6)])
def test_error_comes_before_nan(flag, nan, status):
    from kore_gb300 import _lib
    assert _lib.load().kore_outcome(flag, nan) == status
