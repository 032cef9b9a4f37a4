"""The matrix maximum that scales an exact product's operands, for thin and ragged
operands and wherever the largest element lies."""
import ctypes

import numpy as np
import pytest

from bem_gb300 import _lib, api

pytestmark = pytest.mark.gpu


# rows and columns around the powers of two that divide a 2048-element chunk
@pytest.mark.parametrize("m,k", [(1, 1), (1, 2049), (2, 2047), (3, 700), (31, 65), (64, 33), (255, 9), (257, 5),
                                 (1023, 3), (1025, 3), (2047, 2), (2049, 2), (4100, 1)])
def test_largest_element_anywhere(m, k):
    """One element 2^600 times the others, in A and then in B.  A scale taken without it would
    leave FP32's range (not finite).  With it the others are flushed in its block and are below
    2^-500 of its products elsewhere, so every product is the big element's, to the slices'
    rounding of 2^-40 and the FP32 sums' 2^-40 of it."""
    import torch
    L = _lib.load()
    ctx = api.default_context()
    rng = np.random.default_rng(m + 5 * k)
    for r, c in {(0, 0), (m - 1, 0), (0, k - 1), (m - 1, k - 1), (m // 2, k // 2)}:
        big = np.zeros((m, k), dtype=complex)
        big[r, c] = 2.0 ** 600 * (1 - 0.75j)
        big += rng.standard_normal((m, k)) + 1j * rng.standard_normal((m, k))
        thin = rng.standard_normal((k, 3)) + 1j * rng.standard_normal((k, 3))
        for A, B in ((big, thin), (np.ascontiguousarray(thin.T), np.ascontiguousarray(big.T))):
            mm, kk, nn = A.shape[0], A.shape[1], B.shape[1]
            dA, dB = (torch.from_numpy(np.ascontiguousarray(x.T)).cuda() for x in (A, B))
            dC = torch.zeros((nn, mm), dtype=torch.complex128, device="cuda")
            torch.cuda.synchronize()
            rc = L.bemgpu_zgemm_exact(ctx.handle, mm, nn, kk, ctypes.c_void_p(dA.data_ptr()), mm,
                                      ctypes.c_void_p(dB.data_ptr()), kk, ctypes.c_void_p(dC.data_ptr()), mm, 0, 5)
            assert rc == _lib.OK, L.bemgpu_ctx_last_error(ctx.handle)
            C, ref = dC.cpu().numpy().T, A @ B
            assert np.isfinite(C).all()
            assert np.abs(C - ref).max() < 2.0 ** -36 * 2.0 ** 600 * np.abs(thin).max()
