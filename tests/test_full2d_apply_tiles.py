"""The Full-2D apply where its kernels cut their work: rho_x and columns around whole warps and tiles, rho_y tables that
fit and do not fit the shared memory, every number of local nodes, many quadrature points.

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
