"""The 5 x 5 exact product's 128 x 96 tiles against its 128 x 64 ones at the edges of the 96 columns."""
import ctypes

import numpy as np
import pytest

from bem_gb300 import _lib, api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(65, 95, 64), (64, 96, 65), (130, 97, 300), (33, 191, 129), (200, 193, 1000),
                                   (1, 385, 17)])
@pytest.mark.parametrize("accumulate", [0, 1])
def test_same_sums_on_both_tiles(m, n, k, accumulate):
    """Both keep a sum for each level and add a block's products to it in the same order: the same bits."""
    import torch
    L = _lib.load()
    ctx = api.default_context()
    gen = torch.Generator(device="cuda").manual_seed(m + 3 * n + 5 * k)

    def draw(r, c):
        return torch.randn((c, r), generator=gen, dtype=torch.complex128, device="cuda")

    A, B, C = draw(m, k), draw(k, n), draw(m, n)

    def run(tiles):
        assert L.bemgpu_ctx_set_tuning(ctx.handle, _lib.TUNE_EX_WIDE, tiles) == _lib.OK
        out = C.clone()
        torch.cuda.synchronize()
        rc = L.bemgpu_zgemm_exact(ctx.handle, m, n, k, ctypes.c_void_p(A.data_ptr()), m, ctypes.c_void_p(B.data_ptr()), k,
                                  ctypes.c_void_p(out.data_ptr()), m, accumulate, 5)
        assert rc == _lib.OK, L.bemgpu_ctx_last_error(ctx.handle)
        return out.cpu().numpy()

    try:
        narrow, wide = run(0), run(2)
    finally:
        L.bemgpu_ctx_set_tuning(ctx.handle, _lib.TUNE_EX_WIDE, 1)
    assert np.array_equal(narrow, wide)
