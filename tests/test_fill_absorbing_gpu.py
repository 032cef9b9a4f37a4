"""FP64 fills between bodies many absorption lengths apart, entry by entry against the oracle."""
import numpy as np
import pytest

from bem_gb300 import _lib, api, mesh
from oracle import oracle
from tests.cases import row_scaled_err

pytestmark = pytest.mark.gpu


# Im k of 20, 40, 100 over distances of 3 to 5.6: e^-60 to e^-560, within FP64's range
@pytest.mark.parametrize("im_k", [20.0, 40.0, 100.0])
def test_entries_beyond_fp32s_range(im_k):
    """e^{-Im k R} is off by Im k R roundings, 560 x 2^-53 = 6e-14 of each entry: the fill's
    bar of 1e-10 of a row's largest holds for rows that are that small as a whole."""
    v, t = mesh.cube(1.0, 1)
    b2 = mesh.Body.from_mesh(v, t)
    b1 = b2.translated(mesh.gap_translation(v, v, 3.0))
    d = api.FixedLorentz(*api.SIC_CONFIG)
    _, s, tt = api.parseShapes(b1, b2, d, d)
    xyz, tris, rwg, ns = mesh.two_body(b1, b2)
    k = 0.7 + 1j * im_k
    eps, omega = (k / 0.5) ** 2, 0.5
    ref = oracle.zts(xyz, tris, rwg[:ns], rwg[ns:], eps, 1 + 0j, omega)
    assert np.abs(ref).max(axis=1).min() > 0
    Z = api.Zts(s, tt, api.GreensFunction(eps, 1.0, omega, False), precision=_lib.PREC_FP64)
    assert row_scaled_err(Z, ref) < 1e-10
