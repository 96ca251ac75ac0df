"""Inner products of the Full-2D inner solve: odd numbers of unknowns, fewer unknowns
than one block takes, several elements per thread, steps inside and past groups of four vectors, FP32 and FP16 basis.

The mixed solve must meet its tolerance by the FP64 residual formed here (the operator's own rounding, 1e-12 of |b|
at most, is allowed on top), within twice the FP64 solver's iterations plus the refinements' restarts: wrong
coefficients or norms leave the inner solves without an orthogonal basis.
"""
import numpy as np
import pytest

from test_full2d import det_vec, make_mat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("basis16", [False, True])
@pytest.mark.parametrize("restart", [7, 40])
@pytest.mark.parametrize("cfg", [dict(yb="zero-inflow", nex=3, ney=1, nrx=9, nry=3), dict(nex=4, nrx=9, nry=4),
                                 dict(nex=5, nrx=21, nry=5), dict(nex=40, nrx=61, nry=12)])
def test_inner_products(built_lib, cfg, restart, basis16):
    from real_space_dg_gb300.full2d import Full2DOperator
    mat, V = make_mat(**cfg)
    with Full2DOperator(mat, V) as op:
        op.set_preconditioner()
        b = det_vec(op.n)
        st, ref, _ = op.solve(b, tol=1e-9, maxit=600, restart=restart, mixed=False)
        assert st == 0
        st, info, x = op.solve(b, tol=1e-9, maxit=600, restart=restart, mixed=True, inner_basis_fp16=basis16)
        r = b - op.apply(x)
        assert st == 0 and np.linalg.norm(r) <= 1.001e-9 * np.linalg.norm(b)
        assert info["iterations"] <= 2 * ref["iterations"] + 40, (info, ref)
