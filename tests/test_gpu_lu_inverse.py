"""The camera blocks' inverse by a warp (the PCG set-up) equals the one by a
thread to the bit, at every size, with and without exchanged pivots."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("np_", range(1, 10))
def test_warp_equals_thread(np_):
    import rpba_b200 as rb
    rng = np.random.default_rng(np_)
    n = 2048
    A = rng.normal(size=(n, 9, 9)) * 10.0 ** rng.uniform(-6, 6, size=(n, 9, 1))
    A[n // 2:] = A[n // 2:] @ A[n // 2:].transpose(0, 2, 1) + 1e-2 * np.eye(9)
    A[0] = np.eye(9)[::-1]  # every pivot exchanged, ties with zeros
    A[1] = np.where(np.eye(9) > 0, 2.0, 1.0)  # equal candidates
    if np_ < 9:
        A[0, :np_, :np_] = np.eye(np_)[::-1]
    t, w = np.full_like(A, np.nan), np.full_like(A, np.nan)
    dp = C.POINTER(C.c_double)
    st = rb.load().rpba_debug_lu_inverse(A.ctypes.data_as(dp), n, np_, t.ctypes.data_as(dp), w.ctypes.data_as(dp), 0)
    assert st == 0
    assert np.isfinite(t).all()
    # (by value: the padding's zeros may differ in sign)
    assert np.array_equal(t, w)
    # the well-conditioned one against the closed form: (I + 1 1^T)^-1 = I - 1 1^T / (1 + np)
    ref = np.eye(np_) - 1.0 / (1 + np_)
    assert np.abs(t[1, :np_, :np_] - ref).max() <= 1e-14
