"""The fill's routes against the oracle: the near pairs' series of few and of
more powers and their direct evaluation (chosen by |k| R), lossless and lossy
media, every far rule, and triangle counts around the far kernel's 32 x 32
blocks, in FP64 and in double-float.

Tolerances: FP64 entries within 1e-10 of their row's scale (the fill's bar);
double-float ones within 1e-11, two hundred roundings of 2^-47 with the up to
~10x cancellation of a row's entries."""
import numpy as np
import pytest

from bem_gb300 import _lib, api, mesh
from oracle import oracle
from tests.cases import row_scaled_err

pytestmark = pytest.mark.gpu
TOL = {_lib.PREC_FP64: 1e-10, _lib.PREC_MIXED_LA: 1e-11}


def _bodies(n1, n2, gap):
    v2, t2 = mesh.cube(1.0, n2)
    v1, t1 = mesh.cube(1.0, n1)
    b2 = mesh.Body.from_mesh(v2, t2)
    return mesh.Body.from_mesh(v1 + mesh.gap_translation(v1, v2, gap), t1), b2


def _check(n1, n2, gap, eps, omega, external, far=None):
    b1, b2 = _bodies(n1, n2, gap)
    d = api.FixedLorentz(*api.SIC_CONFIG)
    top, s, t = api.parseShapes(b1, b2, d, d)
    xyz, tris, rwg, ns = mesh.two_body(b1, b2)
    o = api.Options()
    if far is not None:
        o.farThresh6, o.farThresh10, o.farThresh15, o.farThresh21 = far
    g = api.GreensFunction(eps, 1.0, omega, external)
    for prec, tol in TOL.items():
        for rows, cols, a, b in ((top, top, rwg, rwg), (s, t, rwg[:ns], rwg[ns:])):
            ref = oracle.zts(xyz, tris, a, b, complex(eps), 1 + 0j, omega, **({} if far is None else {"far": far}))
            assert row_scaled_err(api.Zts(rows, cols, g, o, precision=prec), ref) < tol, (prec, rows.rwgs, cols.rwgs)


# cubes of 2 x 2 squares: edges up to 0.707, so |k| R <= 1.414 |k|; the series
# kinds end at |k| R = 0.47 and 1.1
@pytest.mark.parametrize("kr", [0.02, 0.469, 0.471, 1.09, 1.11, 6.0])
@pytest.mark.parametrize("eps", [1.0, 1.0 + 0.4j, -1.0 + 0.05j])
def test_near_kinds(kr, eps):
    k = kr / (2.0 * 0.5 * 2.0 ** 0.5)
    omega = k / abs(np.sqrt(complex(eps)))
    _check(2, 2, 0.2, eps, omega, eps == 1.0)


# thresholds that make one far rule the rule of (nearly) every pair
@pytest.mark.parametrize("far", [(1e9, 8.0, 4.0, 2.0), (0.0, 1e9, 4.0, 2.0), (0.0, 0.0, 1e9, 2.0), (0.0, 0.0, 0.0, 1e9),
                                 (0.0, 0.0, 0.0, 0.0), (1.0, 0.5, 0.25, 0.1)])
@pytest.mark.parametrize("eps", [1.0, 2.0 + 0.5j])
def test_far_rules(far, eps):
    _check(1, 2, 0.05, eps, 0.5, eps == 1.0, far)


# 12 and 48 triangles (below, above and between multiples of 32), a gap far
# below the edges (36-point pairs) and one above them
@pytest.mark.parametrize("n1,n2,gap", [(1, 1, 0.01), (1, 2, 0.01), (2, 1, 3.0), (2, 3, 0.03)])
def test_far_blocks(n1, n2, gap):
    _check(n1, n2, gap, 1.0, 0.5, True)


@pytest.mark.parametrize("eV", [0.0905, 0.0983, 0.118])
@pytest.mark.parametrize("precision", [_lib.PREC_FP64, _lib.PREC_MIXED_LA])
def test_shared_near_pairs_of_a_solve(eV, precision):
    """A solve's interior near pairs ride on the exterior's (or, at resonance,
    run directly): the batch of two frequencies and the oracle agree."""
    b1, b2 = _bodies(2, 3, 0.15)
    d = api.FixedLorentz(*api.SIC_CONFIG)
    top, s, t = api.parseShapes(b1, b2, d, d)
    xyz, tris, rwg, ns = mesh.two_body(b1, b2)
    jobs = [(1e-6, f, 300.0, 0.0, top, s, t) for f in (eV, 0.1)]
    P = api.CalcHeatTransferBatch(jobs, precision=precision)
    for (a, f, T1, T2, *_), p in zip(jobs, P):
        eps = d.eps(f)
        ref = oracle.calc_heat_transfer(a, f, T1, T2, xyz, tris, rwg, ns, eps, eps)
        assert abs(p / ref - 1) < (1e-8 if precision == _lib.PREC_FP64 else 1e-6)
