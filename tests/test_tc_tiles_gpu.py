"""The persistent tensor-core complex64 GEMM over its tile widths: one and several tiles per
CTA, ragged edges, few K steps and many."""
import ctypes

import pytest

from bem_gb300 import _lib, api

pytestmark = pytest.mark.gpu


# 128 x 64 tiles, 128 x 128 ones, 128 x 256 ones; the largest of each on more than one round
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (64, 64, 16), (65, 63, 33), (300, 600, 64), (1152, 1151, 130),
                                   (1153, 1152, 1100), (2049, 2047, 250), (4001, 2003, 520), (3841, 3839, 256)])
@pytest.mark.parametrize("accumulate", [0, 1])
@pytest.mark.parametrize("wide_a", [True, False])
def test_cgemm_tc_tiles_exact_on_integers(m, n, k, accumulate, wide_a):
    """One operand holds integers below 2^11 (two bf16 slices), the other -1, 0 or 1, C
    integers below 2^11: every partial sum is an integer below 2 x 1100 x 2^11 + 2^11 <
    2^23, so each FP32 add is exact and so is the result."""
    import torch
    L = _lib.load()
    ctx = api.default_context()
    gen = torch.Generator(device="cuda").manual_seed(m + 3 * n + 5 * k)

    def draw(r, c, top):  # column-major r x c
        return torch.randint(-top, top + 1, (c, r, 2), generator=gen, device="cuda").to(torch.float32)

    A, B, C = draw(m, k, 2047 if wide_a else 1), draw(k, n, 1 if wide_a else 2047), draw(m, n, 2047)
    out = C.clone()
    torch.cuda.synchronize()
    rc = L.bemgpu_cgemm(ctx.handle, m, n, k, ctypes.c_void_p(A.data_ptr()), m, ctypes.c_void_p(B.data_ptr()), k,
                        ctypes.c_void_p(out.data_ptr()), m, accumulate, 1)
    assert rc == _lib.OK, L.bemgpu_ctx_last_error(ctx.handle)
    Z = [torch.view_as_complex(x).to(torch.complex128) for x in (A, B, C)]
    want = Z[1] @ Z[0] + (Z[2] if accumulate else 0)
    assert torch.equal(torch.view_as_complex(out).to(torch.complex128), want)
