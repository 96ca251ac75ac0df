"""A problem's bits do not depend on the batch it is solved in: the pieces of the Gram-Schmidt sums, the preconditioner's
scan, the transforms' tiles and the launch shapes follow from one problem's size alone."""
import numpy as np
import pytest

from conftest import small_rtd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,n_el,nk,order,batch", [
    ("fp64", 12, 32, 2, 40), ("fp64", 40, 65, 2, 9), ("fp64", 120, 256, 3, 3), ("mixed", 12, 64, 1, 70),
    ("mixed", 60, 128, 2, 19), ("mixed", 90, 256, 3, 17), ("mixed", 140, 256, 3, 6)])
def test_alone_and_in_a_batch(built_lib, precision, n_el, nk, order, batch):
    from real_space_dg_gb300 import Problem1D
    spec, mat, E, efl, efr, m = small_rtd(n_el=n_el, nk=nk, order=order, bias=0.05)
    kw = dict(n_el=n_el, n_local=order + 1, nk=nk, l_xi=spec.l_xi_m, precision=precision)
    rng = np.random.default_rng(0)
    out = []
    for B in (batch, 1):
        with Problem1D(batch=B, **kw) as P:
            for b in range(B):
                # the problem that is compared is the batch's last one
                P.set_potential(b, mat["x"], E * (1 + 0.02 * (B - 1 - b)), m, spec.m_rel, spec.temp_k, efl, efr)
            r = np.zeros((B, P.N), dtype=complex)
            r[-1] = rng.normal(size=P.N) + 1j * rng.normal(size=P.N) if not out else out[0][0]
            P.set_launch_shapes(kline_chunk=max(1, n_el // 30))
            z = P.precondition(r).reshape(B, -1)[-1].copy()
            st, info = P.solve(tol=1e-9, maxit=60)
            assert st == 0
            out.append((r[-1], z, P.rho(B - 1), info[-1]["iterations"]))
    (_, z0, rho0, it0), (_, z1, rho1, it1) = out
    assert np.array_equal(z0, z1)
    assert it0 == it1 and np.array_equal(rho0, rho1)
