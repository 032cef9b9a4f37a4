"""The 128 x 128-tile exact products (5 x 5 and 4 x 4 slices) against the 128 x 64-tile ones
and a complex128 product, at the edges of tiles and exponent blocks."""
import ctypes

import numpy as np
import pytest

from bem_gb300 import _lib, api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (63, 127, 63), (64, 128, 64), (65, 129, 65), (129, 70, 193),
                                   (200, 300, 1000)])
@pytest.mark.parametrize("slices", [4, 5])
def test_wide_tiles_agree_with_narrow_ones_and_with_complex128(slices, m, n, k):
    """Both keep every product of a level below the number of slices.  Against
    complex128 they differ by the dropped levels and the slices' rounding: at most
    slices + 2 products of 2^(-8 slices) of the block maxima's product, below
    2^(4 - 8 slices).  Against each other by FP32 sums of the levels that only one of them
    sums exactly: level 2 for 4 x 4 (2^-16 of the maxima's product, rounded at 2^-24
    of that: 2^-38 for a few roundings of the largest partial sum), the joint
    or separate sums of levels 3 and 4 for 5 x 5 (2^-46, likewise)."""
    import torch
    L = _lib.load()
    ctx = api.default_context()
    rng = np.random.default_rng(m + 7 * n + 31 * k + slices)
    A = (rng.standard_normal((m, k)) + 1j * rng.standard_normal((m, k))) * np.exp(rng.uniform(-3, 3, (m, 1)))
    B = rng.standard_normal((k, n)) + 1j * rng.standard_normal((k, n))
    scale = k * np.outer(np.abs(A).max(axis=1), np.abs(B).max(axis=0))
    dA = torch.from_numpy(np.ascontiguousarray(A.T)).cuda()
    dB = torch.from_numpy(np.ascontiguousarray(B.T)).cuda()

    def run(tiles):
        assert L.bemgpu_ctx_set_tuning(ctx.handle, _lib.TUNE_EX_WIDE, tiles) == _lib.OK
        dC = torch.zeros((n, m), dtype=torch.complex128, device="cuda")
        torch.cuda.synchronize()
        rc = L.bemgpu_zgemm_exact(ctx.handle, m, n, k, ctypes.c_void_p(dA.data_ptr()), m,
                                  ctypes.c_void_p(dB.data_ptr()), k, ctypes.c_void_p(dC.data_ptr()), m, 0, slices)
        assert rc == _lib.OK, L.bemgpu_ctx_last_error(ctx.handle)
        return dC.cpu().numpy().T

    try:
        narrow, wide = run(0), run(2)
    finally:
        L.bemgpu_ctx_set_tuning(ctx.handle, _lib.TUNE_EX_WIDE, 1)
    assert np.max(np.abs(wide - narrow) / scale) < 2.0 ** (-36 if slices == 4 else -44)
    assert np.max(np.abs(wide - A @ B) / scale) < 2.0 ** (4 - 8 * slices)
