"""The quantized B operand: B is replaced by exactly the values that its three slices hold."""
import ctypes

import numpy as np
import pytest

from bem_gb300 import _lib, api

pytestmark = pytest.mark.gpu

BITS, BLOCK = 24, 64


def quantized(B):
    """Block fixed point over 64 complex rows of a column: the block's largest exponent E (|re|,
    |im| < 2^E), values rounded to multiples of 2^(E - 24), halves away from zero; subnormal
    inputs, and blocks below 2^-80 of the matrix's largest exponent, are zero."""
    out = np.zeros_like(B)
    tiny = np.finfo(float).tiny

    def mag(x):
        a = np.maximum(np.abs(x.real), np.abs(x.imag))
        return np.where(a < tiny, 0.0, a)

    top = np.frexp(mag(B).max())[1]
    for r in range(0, B.shape[0], BLOCK):
        for c in range(B.shape[1]):
            x = B[r:r + BLOCK, c]
            m = mag(x).max()
            E = np.frexp(m)[1]
            if m == 0.0 or E - top < -80:
                continue
            parts = []
            for p in (x.real, x.imag):
                v = np.where(np.abs(p) < tiny, 0.0, np.ldexp(np.abs(p), BITS - E))
                n = np.floor(v) + (v - np.floor(v) >= 0.5)
                parts.append(np.copysign(np.ldexp(n, E - BITS), p) * (n > 0))
            out[r:r + BLOCK, c] = parts[0] + 1j * parts[1]
    return out


# ordinary values; near FP64's lower end, where the results leave the normal numbers; near its
# upper end; and blocks far below the largest one, the last of them flushed
@pytest.mark.parametrize("scale,spread", [(0, 0), (-1010, 0), (1020, 0), (0, 20), (-960, 20)])
@pytest.mark.parametrize("n,k", [(1, 1), (3, 64), (5, 65), (7, 300)])
def test_quantized_operand_is_the_slices_value(n, k, scale, spread):
    import torch
    L = _lib.load()
    ctx = api.default_context()
    rng = np.random.default_rng(n + k + spread)
    B = rng.uniform(-1, 1, (k, n)) + 1j * rng.uniform(-1, 1, (k, n))
    B = B * 2.0 ** (-spread * (np.arange(k) // BLOCK))[:, None]
    B = np.ldexp(B.real, scale) + 1j * np.ldexp(B.imag, scale)
    B[rng.integers(k, size=2), rng.integers(n, size=2)] = 0
    m = 2
    dA = torch.ones((k, m), dtype=torch.complex128, device="cuda")
    dB = torch.from_numpy(np.ascontiguousarray(B.T)).cuda()
    dC = torch.zeros((n, m), dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()
    rc = L.bemgpu_zgemm_exact_quantized(ctx.handle, m, n, k, ctypes.c_void_p(dA.data_ptr()), m,
                                        ctypes.c_void_p(dB.data_ptr()), k, ctypes.c_void_p(dC.data_ptr()), m, 0)
    assert rc == _lib.OK, L.bemgpu_ctx_last_error(ctx.handle)
    assert np.array_equal(dB.cpu().numpy().T, quantized(B))
