"""The Full-2D preconditioner where its kernels cut their work, against the oracle's line-transverse inverse."""
import pytest

from oracle import full2d as F2
from test_full2d import det_vec, make_mat, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cfg", [
    dict(nex=8, nrx=9, nry=4), dict(nex=17, nkx=2, nrx=33, nry=4), dict(nex=70, nkx=4, nky=2, nrx=8, nry=4),
    dict(nex=11, nrx=64, nry=5, yb="zero-inflow"), dict(nex=23, nky=4, ney=3, nrx=10, nry=3, yb="specular")])
def test_preconditioner_at_tile_edges(built_lib, cfg):
    """Two and more chunks of a line, ragged ones, blocks of lines and of X dofs cut by the end, an odd transverse
    block, columns that do not fill a tile: FP64 by mode and with rho_x fastest (tensor cores) to 1e-12, FP32 to the
    single-precision rounding of an approximate inverse (2e-5), as for the other shapes."""
    from real_space_dg_gb300.full2d import Full2DOperator
    mat, V = make_mat(**cfg)
    p, parts, dd = F2.system(mat, V)
    ref = F2.line_transverse(mat, p, V, dd)
    r = det_vec(p["nTotal"])
    want = F2.line_transverse_apply(p, ref, r)
    for tc, fp32, tol in ((False, False, 1e-12), (True, False, 1e-12), (False, True, 2e-5)):
        with Full2DOperator(mat, V, tensor_cores=tc) as op:
            op.set_preconditioner(fp32=fp32)
            assert rel(op.precondition(r), want) < tol, (tc, fp32)
