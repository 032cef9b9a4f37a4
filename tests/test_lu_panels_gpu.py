"""Solves whose sizes leave remainders of every blocking of the LU (sub-panels
of 8 and 32 columns, panels of 64 and 128, pairs of panels, clusters of 1 to 16
CTAs of 32 rows), in FP64 and on both mixed factorizations, against the oracle:
FP64 within 1e-8, mixed within 1e-6 (the solves' own bounds)."""
import pytest

from bem_gb300 import _lib, api, mesh
from oracle import oracle

pytestmark = pytest.mark.gpu


# cubes of k x k squares have 18 k^2 RWGs: N = 72, 180, 360, 468, 612, 1152
@pytest.mark.parametrize("n1,n2", [(1, 1), (1, 2), (3, 1), (2, 3), (1, 4), (4, 4)])
@pytest.mark.parametrize("how", ["fp64", "complex64", "fp64class"])
def test_remainders(n1, n2, how):
    v1, t1 = mesh.cube(1.0, n1)
    v2, t2 = mesh.cube(1.0, n2)
    b1, b2 = mesh.Body.from_mesh(v1 + mesh.gap_translation(v1, v2, 0.1), t1), mesh.Body.from_mesh(v2, t2)
    d = api.FixedLorentz(*api.SIC_CONFIG)
    ctx = api.Context(0)
    ctx.set_solver({"fp64": 0, "complex64": 1, "fp64class": 2}[how])
    top, s, t = api.parseShapes(b1, b2, d, d, ctx)
    precision = _lib.PREC_FP64 if how == "fp64" else _lib.PREC_MIXED_LA
    xyz, tris, rwg, ns = mesh.two_body(b1, b2)
    eps = d.eps(0.105)
    ref = oracle.calc_heat_transfer(1e-6, 0.105, 300.0, 0.0, xyz, tris, rwg, ns, eps, eps)
    P = api.CalcHeatTransfer(1e-6, 0.105, 300.0, 0.0, top, s, t, precision=precision)
    assert abs(P / ref - 1) < (1e-8 if how == "fp64" else 1e-6)
    # the same panels with fewer CTAs: the rows' split changes no result
    L = _lib.load()
    for cap in (1, 3):
        assert L.bemgpu_ctx_set_tuning(ctx.handle, _lib.TUNE_PANEL_CTAS, cap) == _lib.OK
        assert api.CalcHeatTransfer(1e-6, 0.105, 300.0, 0.0, top, s, t, precision=precision) == P
