"""The FMA-pipe complex GEMM over the tiles it chooses from."""
import ctypes

import numpy as np
import pytest

from bem_gb300 import _lib, api

pytestmark = pytest.mark.gpu


# 32 x 32, 64 x 64 and 128 x 64 tiles (by their waves on the GPU's SMs), each with edges
# inside a tile, and K of one, less than one and several steps; more columns than one
# launch covers
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (31, 33, 15), (33, 32, 17), (129, 65, 16), (700, 500, 33), (769, 641, 7),
                                   (2049, 1025, 24), (2500, 1300, 9), (2, 1048600, 3)])
@pytest.mark.parametrize("accumulate", [0, 1])
def test_cgemm_fma_tiles(m, n, k, accumulate):
    """A sum of k complex products in FP32 is off by at most (2 k + 2) roundings of the sum of
    the magnitudes |re| and |im| products, which |A| |B| bounds up to a factor of 2."""
    import torch
    L = _lib.load()
    ctx = api.default_context()
    rng = np.random.default_rng(m + n + k)

    def draw(r, c):
        return (rng.standard_normal((r, c)) + 1j * rng.standard_normal((r, c))).astype(np.complex64)

    A, B, C = draw(m, k), draw(k, n), draw(m, n)
    dA, dB, dC = (torch.from_numpy(np.ascontiguousarray(x.T)).cuda() for x in (A, B, C))
    torch.cuda.synchronize()
    rc = L.bemgpu_cgemm(ctx.handle, m, n, k, ctypes.c_void_p(dA.data_ptr()), m, ctypes.c_void_p(dB.data_ptr()), k,
                        ctypes.c_void_p(dC.data_ptr()), m, accumulate, 2)
    assert rc == _lib.OK, L.bemgpu_ctx_last_error(ctx.handle)
    want = A.astype(np.complex128) @ B.astype(np.complex128) + (C if accumulate else 0)
    bound = 2 * (2 * k + 2) * 2.0 ** -24 * (np.abs(A).astype(float) @ np.abs(B).astype(float) + np.abs(C))
    assert np.all(np.abs(dC.cpu().numpy().T - want) <= bound)
