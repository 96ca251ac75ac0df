"""Handles of different shapes used in turn: what one sets up (limits of shared memory belong to the kernels) does not
take anything from the other."""
import numpy as np
import pytest

from test_full2d import det_vec, make_mat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fp32", [False, True])
def test_full2d(built_lib, fp32):
    from real_space_dg_gb300.full2d import Full2DOperator
    (ma, Va), (mb, Vb) = make_mat(nry=16), make_mat(nry=4)
    with Full2DOperator(ma, Va) as a, Full2DOperator(mb, Vb) as b:
        a.set_preconditioner(fp32=fp32)
        r = det_vec(a.n)
        want = a.precondition(r)
        b.set_preconditioner(fp32=fp32)
        b.precondition(det_vec(b.n))
        assert np.array_equal(a.precondition(r), want)


def test_full2d_wide_axis(built_lib):
    """The rho_x factors' columns beyond 48 KB in FP64."""
    from real_space_dg_gb300.full2d import Full2DOperator
    (ma, Va), (mb, Vb) = make_mat(nrx=500, nry=4, nex=3), make_mat(nrx=360, nry=4, nex=3)
    with Full2DOperator(ma, Va) as a:
        x = det_vec(a.n)
        want = a.apply(x)
        with Full2DOperator(mb, Vb) as b:
            b.apply(det_vec(b.n))
            assert np.array_equal(a.apply(x), want)


def test_subbands(built_lib):
    from real_space_dg_gb300.subbands import SubbandSolver
    rng = np.random.default_rng(0)
    data = [(rng.uniform(0.2, 0.5, (1, 3, ny)), rng.uniform(0.0, 0.3, (3, ny))) for ny in (1024, 400)]
    with SubbandSolver(1, 3, 1024, 4) as a:
        want = a.solve(*data[0], 0.1)
        with SubbandSolver(1, 3, 400, 4) as b:
            b.solve(*data[1], 0.1)
            got = a.solve(*data[0], 0.1)
    assert all(np.array_equal(g, w) for g, w in zip(got, want))
