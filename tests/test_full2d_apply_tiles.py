"""The Full-2D apply where its kernels cut their work: rho_x around the 31 cells of a warp, fewer and more rows of
cells than one warp takes, every number of local nodes, more quadrature points than one launch stages.

Against the oracle's assembled operator, 1e-12 relative as for the other shapes (the same sums in another order).
"""
import pytest

from oracle import full2d as F2
from test_full2d import det_vec, make_mat, oracle_apply, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cfg", [
    dict(nrx=30, nry=4), dict(nrx=31, nry=5), dict(nrx=32, nry=7, yb="zero-inflow", fx="rusanov", fy="central"),
    dict(nrx=62, nry=4, nex=3), dict(nrx=63, nry=13, nex=2, yb="specular"), dict(nrx=7, nry=40, nex=2),
    dict(nkx=2, nky=2, nrx=9, nry=4), dict(nkx=4, nky=3, nrx=9, nry=4), dict(nkx=2, nky=3, nrx=33, nry=6),
    dict(nkx=4, nky=2, nrx=9, nry=6), dict(nkx=4, nky=4, nex=2, nrx=12, nry=4), dict(nex=2, nq=17, nrx=9, nry=4)])
def test_apply_at_tile_edges(built_lib, cfg):
    from real_space_dg_gb300.full2d import Full2DOperator
    mat, V = make_mat(**cfg)
    p, parts, dd = F2.system(mat, V)
    u = det_vec(p["nTotal"])
    want = oracle_apply(mat, p, parts, dd, u)
    for tc in (False, True):
        with Full2DOperator(mat, V, tensor_cores=tc) as op:
            assert rel(op.apply(u), want) < 1e-12


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
