"""Flow integrals at odd and even radial truncations, around a warp and a CTA of point
pairs, and for odd numbers of vectors, against the reference's formulas (oracle)."""
import numpy as np
import pytest

from oracle.diag_ref import flow_l

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,nvec", [(2, 1), (3, 2), (24, 3), (63, 1), (64, 2), (65, 3), (512, 2), (515, 1), (1027, 3)])
def test_flow_integrals_match_oracle(gpu_lib, N, nvec):
    from kore_gb300.diagnostics import flow_integrals
    m, lmax, ricb = 2, 5, 0.35
    rng = np.random.default_rng(N)
    nb = lmax - m + 1
    x = rng.standard_normal((nb, N, nvec)) + 1j * rng.standard_normal((nb, N, nvec))
    x *= np.exp(-0.1 * np.arange(N))[None, :, None]
    X = x.reshape(nb * N, nvec)
    per, degrees = flow_integrals(X, m, 1, lmax, N, ricb)
    for v in range(nvec):
        for b, l in enumerate(degrees):
            ref = np.array(flow_l(int(l), X[b * N:(b + 1) * N, v], b >= nb // 2, N, ricb)[:3])
            # sums of N terms of sums of N terms (each u sqrt(N)) of coefficients that decay,
            # third derivatives growing as k^6 / 15 over their range: 1e-11 as for the
            # reference's own integrals
            assert np.all(np.abs(per[v, b] - ref) <= 1e-11 * np.abs(ref).max() + 1e-300), (v, l, per[v, b], ref)
