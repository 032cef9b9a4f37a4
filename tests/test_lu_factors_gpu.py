"""The LU factorizations by themselves, on matrices whose factors are known exactly: every
value on the way is a small multiple of a power of two, so the factors and the
interchanges have to come out bit for bit, on every route a panel takes (one-row and two-row
clusters, the cooperative grid beyond 16384 rows, and the hand-over between them)."""
import ctypes

import numpy as np
import pytest
import scipy.sparse as sp

from bem_gb300 import _lib, api

pytestmark = pytest.mark.gpu

# C++ entry points of the library (dense.cu)
NAMES = {"c": "_Z10bem_cgetrfP12bemgpu_ctx_sPfliPiS2_P11CUstream_st",
         "z": "_Z10bem_zgetrfP12bemgpu_ctx_sPdliPiS2_P11CUstream_st",
         "zexact": "_Z16bem_zgetrf_exactP12bemgpu_ctx_sPdliPiS2_P11CUstream_st"}
UNITS = np.array([1, 1j, -1, -1j])


def _dense(A, dtype):
    """Column-major on the device: the transpose of the torch tensor."""
    import torch
    A = A.tocoo()
    out = torch.zeros(A.shape[::-1], dtype=dtype, device="cuda")
    out[torch.from_numpy(A.col).long().cuda(), torch.from_numpy(A.row).long().cuda()] = \
        torch.from_numpy(A.data.astype(np.complex128)).to(dtype).cuda()
    return out


def _factor(how, A):
    """A (sparse) -> the packed factors on the device, ipiv, info."""
    import torch
    n = A.shape[0]
    dA = _dense(A, torch.complex64 if how == "c" else torch.complex128)
    ipiv = torch.empty(n, dtype=torch.int32, device="cuda")
    info = torch.empty(1, dtype=torch.int32, device="cuda")
    f = getattr(_lib.load(), NAMES[how])
    f.restype, p = ctypes.c_int, ctypes.c_void_p
    f.argtypes = [p, p, ctypes.c_int64, ctypes.c_int, p, p, p]
    torch.cuda.synchronize()
    rc = f(api.default_context().handle, dA.data_ptr(), n, n, ipiv.data_ptr(), info.data_ptr(), None)
    assert rc == _lib.OK
    torch.cuda.synchronize()
    return dA, ipiv.cpu().numpy(), int(info[0])


def _known_factors(n, rng):
    """L = I + N and U = D + M, N from even columns into odd rows and M from even rows into
    odd columns: N^2 = 0 and (D^-1 M)^2 = 0, so the triangles' inverses are exact too."""
    def pairs():  # an odd index and a smaller even one, each pair once
        odd = 2 * rng.integers(0, max(1, n // 2), 4 * n) + 1
        even = 2 * rng.integers(0, (n + 1) // 2, 4 * n)
        keep = (odd < n) & (even < odd)
        return np.unique(np.stack([odd[keep], even[keep]], axis=1), axis=0).T

    i, j = pairs()
    N = sp.coo_matrix((0.5 * UNITS[rng.integers(0, 4, i.size)], (i, j)), shape=(n, n)).tocsr()
    i, j = pairs()
    M = sp.coo_matrix((UNITS[rng.integers(0, 4, i.size)], (j, i)), shape=(n, n)).tocsr()
    return sp.identity(n, format="csr") + N, sp.diags(4.0 * UNITS[rng.integers(0, 4, n)]).tocsr() + M


@pytest.mark.parametrize("how,n", [("c", 1), ("c", 33), ("c", 500), ("c", 4097), ("c", 8300), ("c", 16640),
                                   ("z", 1), ("z", 65), ("z", 500), ("z", 2049), ("zexact", 1100), ("zexact", 8300),
                                   ("zexact", 16640)])
def test_known_factors(how, n):
    """Rows in random order: the largest of each column is the only one of its size."""
    import torch
    rng = np.random.default_rng(n)
    Lf, U = _known_factors(n, rng)
    A = (Lf @ U).tocsr()
    order = rng.permutation(n)
    got, ipiv, info = _factor(how, A[order])
    assert info == 0
    rows = order.copy()
    for k, p in enumerate(ipiv):
        rows[k], rows[p] = rows[p], rows[k]
    assert np.array_equal(rows, np.arange(n))
    want = _dense((Lf - sp.identity(n, format="csr") + U).tocsr(), got.dtype)
    assert torch.equal(got, want)


@pytest.mark.parametrize("how", ["c", "z", "zexact"])
@pytest.mark.parametrize("power", [6, 11])
def test_first_of_equals(how, power):
    """A Hadamard matrix with its rows turned by units: each column's candidates are of one
    size, the first is the pivot, and there is no interchange."""
    import torch
    n = 2 ** power
    Lf, U = np.ones((1, 1)), np.ones((1, 1))
    for _ in range(power):
        Lf, U = np.kron(Lf, [[1, 0], [1, 1]]), np.kron(U, [[1, 1], [0, -2]])
    r = UNITS[np.random.default_rng(power).integers(0, 4, n)]
    got, ipiv, info = _factor(how, sp.coo_matrix(r[:, None] * (Lf @ U)))
    assert info == 0
    assert np.array_equal(ipiv, np.arange(n))
    want = r[:, None] * (Lf - np.eye(n)) / r[None, :] + r[:, None] * U
    assert torch.equal(got, _dense(sp.coo_matrix(want), got.dtype))


@pytest.mark.parametrize("how", ["c", "z", "zexact"])
def test_pivot_reciprocals_are_rounded_twice(how):
    """2 x 2 blocks [[p, 0], [1, 1]] with p real or imaginary: the multiplier is 1/p as p / |p|^2
    gives it, the square rounded once and the division once."""
    n, real = 512, np.float32 if how == "c" else np.float64
    rng = np.random.default_rng(11)
    p = np.exp(rng.uniform(0.1, 9.0, n // 2)).astype(real)
    turn = UNITS[rng.integers(0, 4, n // 2)]
    i = np.arange(0, n, 2)
    A = sp.coo_matrix((np.concatenate([p * turn, np.ones(n)]),
                       (np.concatenate([i, i + 1, i + 1]), np.concatenate([i, i, i + 1]))), shape=(n, n))
    got, ipiv, info = _factor(how, A)
    assert info == 0 and np.array_equal(ipiv, np.arange(n))
    want = (p / (p * p)).astype(np.float64) * turn.conj()
    assert np.array_equal(got.cpu().numpy().T[i + 1, i], want)
