"""FP64 kernels of the plain form at the sizes where their tiles end."""
import numpy as np
import pytest

from conftest import small_rtd
from oracle import dg1d, krylov

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_el,nk,nxi,order", [
    (1, 8, 8, 1), (2, 15, 15, 1), (3, 16, 17, 2), (3, 17, 18, 1), (5, 31, 40, 3), (2, 63, 63, 2), (3, 64, 66, 1),
    (2, 65, 65, 3), (3, 127, 129, 1), (2, 130, 131, 2)])
def test_paired_transforms(built_lib, n_el, nk, nxi, order):
    """Phi rho and the operator (both transforms) with odd and even Nk and N_xi around the tiles of 8, 16 and 32
    rows and the chunks of 32 pairs.  A sum of nk terms of size |x| / sqrt(L) carries at most nk eps of their
    absolute sum, and the phases k xi (up to pi nk / 2) another pi nk / 2 eps."""
    from real_space_dg_gb300 import Problem1D
    spec, mat, E, efl, efr, m = small_rtd(n_el=n_el, nk=nk, order=order, n_xi=nxi)
    p = dg1d.init_params(mat, efl, efr, E, m)
    rng = np.random.default_rng(nk)
    with Problem1D(n_el=n_el, n_local=order + 1, nk=nk, n_xi=nxi, l_xi=spec.l_xi_m) as P:
        P.set_potential(0, mat["x"], E, m, spec.m_rel, spec.temp_k, efl, efr)
        x = rng.normal(size=P.N) + 1j * rng.normal(size=P.N)
        P.set_rho(0, x)
        X = x.reshape(-1, nk)
        bound = 2.3e-16 * (1 + np.pi / 2) * nk * np.abs(X).sum(1) / np.sqrt(spec.l_xi_m)
        assert np.all(np.abs(P.rho_xi(0) - X @ p["phi"].T) <= bound[:, None])
        want = krylov.Operator1D(mat, p, E).apply(x)
        assert np.linalg.norm(P.apply(x) - want) <= 1e-12 * np.linalg.norm(want)
