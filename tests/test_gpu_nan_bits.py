"""A NaN whose bits are all set (a buffer filled with 0xFF) in a right-hand side is an ordinary
NaN: solves end at once with KORE_ENAN or a NaN in the solution, and the next solve is clean."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KORE_ENAN = 8


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("where", ["one", "all"])
@pytest.mark.parametrize("nshift", [1, 3])
def test_all_bits_set(gpu_lib, case, precision, where, nshift):
    import torch
    from kore_gb300 import Pencil, layout_from_params
    from kore_gb300 import _lib as L
    meta, A, B = case("shell_m1_ek1e-4")
    rng = np.random.default_rng(2)
    n = A.shape[0]
    good = rng.standard_normal((n, nshift)) + 1j * rng.standard_normal((n, nshift))
    bad = good.copy()
    bits = bad.view(np.uint64).reshape(n, -1)
    bits[slice(None) if where == "all" else n // 2] = np.uint64(0xFFFFFFFFFFFFFFFF)
    with Pencil(A, B, layout=layout_from_params(meta)) as p:
        p.factor_shifts(complex(*meta["tau"]) + 0.1j * np.arange(nshift), precision)
        x = p.solve(good)
        with pytest.raises(L.KoreError) as e:
            p.solve(bad)
        assert e.value.status == KORE_ENAN
        np.testing.assert_array_equal(p.solve(good), x)
        if nshift == 1:
            stream = torch.cuda.current_stream().cuda_stream
            b = torch.from_numpy(bad.ravel()).cuda()
            y = torch.zeros_like(b)
            rc = p.lib.kore_solve_dev_noalloc(p._plan, ctypes.c_void_p(b.data_ptr()), ctypes.c_void_p(y.data_ptr()), 0.0,
                                              ctypes.c_void_p(stream))
            torch.cuda.synchronize()
            assert rc == (KORE_ENAN if precision == "mixed" else 0)
            assert rc != 0 or bool(torch.isnan(y.real).any())
