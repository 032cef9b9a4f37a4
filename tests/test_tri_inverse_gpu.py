"""The mixed-precision solve by explicit triangle inverses at sizes around their 64-row blocks."""
import pytest

from bem_gb300 import _lib, api, mesh

pytestmark = pytest.mark.gpu


# N = 120, 300, 480: one block and a ragged one, ragged pairs of blocks, whole pairs
@pytest.mark.parametrize("levels", [(0, 0), (0, 1), (1, 1)])
def test_ragged_triangle_blocks(levels):
    """Wrong inverses would not refine: the solve would escalate, or differ from FP64 by more
    than the 1e-6 that the mixed path keeps to."""
    (v1, t1), (v2, t2) = (mesh.icosphere(1.0, level, jitter=0.02, seed=7 + level) for level in levels)
    b1, b2 = mesh.Body.from_mesh(v1, t1), mesh.Body.from_mesh(v2, t2)
    b1 = b1.translated(mesh.gap_translation(v1, v2, 0.2))
    d = api.FixedLorentz(*api.SIC_CONFIG)
    top, s, t = api.parseShapes(b1, b2, d, d)
    for eV in (0.0983, 0.125):
        info = {}
        P = api.CalcHeatTransfer(1e-6, eV, 300.0, 0.0, top, s, t, precision=_lib.PREC_MIXED_LA, info=info)
        P64 = api.CalcHeatTransfer(1e-6, eV, 300.0, 0.0, top, s, t, precision=_lib.PREC_FP64)
        assert abs(P / P64 - 1) < 1e-6, (levels, eV, P, P64)
        assert info["solver"] == 1 and 1 <= info["refine_iters"] <= 4, info
