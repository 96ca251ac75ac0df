"""Transform and Gram-Schmidt kernels of the 1D path at the sizes where their tiles end."""
import numpy as np
import pytest

from conftest import small_rtd
from oracle import dg1d, krylov

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_el,nk,nxi,order", [
    (2, 8, 8, 1), (2, 15, 15, 1), (3, 16, 17, 2), (3, 17, 18, 1), (5, 31, 40, 3), (2, 63, 63, 2), (3, 64, 66, 1),
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


def _residual(P, rho):
    b = P.rhs()
    return np.linalg.norm(b - P.apply(rho)) / np.linalg.norm(b)


@pytest.mark.parametrize("reorth", [0.0, 1.0, -1.0])
@pytest.mark.parametrize("n_el,nk,order", [(5, 17, 1), (40, 65, 2), (100, 96, 3), (140, 96, 3), (272, 96, 3)])
def test_gram_schmidt_fp64(built_lib, n_el, nk, order, reorth):
    """The FP64 Arnoldi at sizes below one block, with 1, 2, 4 and 8 elements per thread of the multi-dot, with
    one, a tested and two Gram-Schmidt passes: the solution meets the tolerance by its own residual.  The
    residual of the solver and the one formed here differ by the operator's rounding (1e-13 of |b| allowed)."""
    from real_space_dg_gb300 import Problem1D
    spec, mat, E, efl, efr, m = small_rtd(n_el=n_el, nk=nk, order=order, bias=0.05)
    with Problem1D(n_el=n_el, n_local=order + 1, nk=nk, l_xi=spec.l_xi_m, reorth=reorth, restart=37) as P:
        P.set_potential(0, mat["x"], E, m, spec.m_rel, spec.temp_k, efl, efr)
        st, info = P.solve(tol=1e-10, maxit=60)
        assert st == 0 and _residual(P, P.rho(0)) <= 1.001e-10


@pytest.mark.parametrize("basis32", [False, True])
@pytest.mark.parametrize("inner_reorth", [0.0, 0.7, 1.0])
@pytest.mark.parametrize("n_el,nk,order,batch", [(5, 36, 2, 1), (2, 32, 1, 3), (16, 64, 1, 2), (31, 68, 3, 3)])
def test_gram_schmidt_mixed(built_lib, n_el, nk, order, batch, inner_reorth, basis32):
    """The inner FP32 Arnoldi (FP16 and FP32 basis) around its blocks of 512 and 2,048 elements, with one, a tested
    and two passes: every problem of the batch meets the tolerance by its own FP64 residual."""
    from real_space_dg_gb300 import Problem1D
    spec, mat, E, efl, efr, m = small_rtd(n_el=n_el, nk=nk, order=order, bias=0.05)
    with Problem1D(n_el=n_el, n_local=order + 1, nk=nk, l_xi=spec.l_xi_m, batch=batch, precision="mixed",
                   inner_reorth=inner_reorth, inner_basis_fp32=basis32, inner_restart=29) as P:
        for b in range(batch):
            P.set_potential(b, mat["x"], E * (1 + 0.02 * b), m, spec.m_rel, spec.temp_k, efl, efr)
        st, info = P.solve(tol=1e-10, maxit=60)
        rho = np.concatenate([P.rho(b) for b in range(batch)])
        r = (P.rhs() - P.apply(rho)).reshape(batch, -1)
        assert st == 0
        assert np.all(np.linalg.norm(r, axis=1) <= 1.001e-10 * np.linalg.norm(P.rhs().reshape(batch, -1), axis=1))


@pytest.mark.parametrize("n_el,nk,nxi,order,batch", [
    (2, 16, 20, 1, 1), (3, 36, 40, 2, 2), (5, 64, 64, 3, 1), (2, 132, 140, 2, 3), (3, 256, 264, 1, 1),
    (2, 260, 512, 1, 2), (4, 512, 512, 1, 1)])
def test_paired_transforms_on_tensor_cores(built_lib, n_el, nk, nxi, order, batch):
    """The digit-sliced transforms with rows below and above one tile of 128 pairs, padded rows, column tiles cut
    by the end of a problem and of a plane: the operator against the native FP64 kernels.  48-bit digits of the
    largest entry of each column: 2^-47 of |Phi| |x| per pair, sums of up to 512 of them, far below 1e-12 of |A x|."""
    from real_space_dg_gb300 import Problem1D
    spec, mat, E, efl, efr, m = small_rtd(n_el=n_el, nk=nk, order=order, n_xi=nxi)
    rng = np.random.default_rng(nk)
    out = []
    for tc in (False, True):
        with Problem1D(n_el=n_el, n_local=order + 1, nk=nk, n_xi=nxi, l_xi=spec.l_xi_m, batch=batch, fp64_tc=tc) as P:
            for b in range(batch):
                P.set_potential(b, mat["x"], E * (1 + 0.1 * b), m, spec.m_rel, spec.temp_k, efl, efr)
            if not out:
                x = rng.normal(size=P.N * batch) + 1j * rng.normal(size=P.N * batch)
            out.append(P.apply(x).reshape(batch, -1))
    want, got = out
    assert np.all(np.linalg.norm(got - want, axis=1) <= 1e-12 * np.linalg.norm(want, axis=1))


@pytest.mark.parametrize("n_el,nk,order,batch", [(64, 12, 1, 1), (64, 36, 1, 1), (63, 36, 3, 2), (33, 20, 2, 5),
                                                 (33, 44, 2, 5), (8, 64, 2, 1), (2, 12, 1, 3), (2, 32, 1, 3),
                                                 (257, 40, 1, 1)])
def test_kline_sweep_in_one_launch(built_lib, n_el, nk, order, batch):
    """Chunk lengths on both sides of the limit of the one-launch sweep, ragged last chunks, padded lines and
    warps.  FP64 against the sequential sweep: sums of n_el contracting maps, 1e-12 as for the two-launch form.
    Mixed (Nk of 32 and more): the chunk length changes FP32 rounding only, so the iterations stay within a quarter
    (plus two; a wrong map doubles them) and the solution meets the tolerance by its own residual."""
    from real_space_dg_gb300 import Problem1D
    spec, mat, E, efl, efr, m = small_rtd(n_el=n_el, nk=nk, order=order, bias=0.05)
    Ls = [L for L in (1, 2, 3, 5, 8, 10, 16, 17) if L <= n_el and -(-n_el // L) <= 64]
    op = krylov.Operator1D(mat, dg1d.init_params(mat, efl, efr, E, m), E)
    ref = krylov.KLinePreconditioner(op, use_drift_diag=False)
    rng = np.random.default_rng(nk)
    kw = dict(n_el=n_el, n_local=order + 1, nk=nk, l_xi=spec.l_xi_m, batch=batch)
    with Problem1D(**kw) as P:
        for b in range(batch):
            P.set_potential(b, mat["x"], E, m, spec.m_rel, spec.temp_k, efl, efr)
        x = rng.normal(size=(batch, P.N)) + 1j * rng.normal(size=(batch, P.N))
        want = np.concatenate([ref.apply(v) for v in x])
        for L in Ls:
            P.set_launch_shapes(kline_chunk=L)
            got = P.precondition(x)
            assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want), L
    if nk < 32:
        return
    its = []
    with Problem1D(precision="mixed", **kw) as P:
        for b in range(batch):
            P.set_potential(b, mat["x"], E * (1 + 0.02 * b), m, spec.m_rel, spec.temp_k, efl, efr)
        rhs = P.rhs().reshape(batch, -1)
        for L in Ls:
            P.set_launch_shapes(kline_chunk=L)
            st, info = P.solve(tol=1e-10, maxit=60)
            assert st == 0 and P.runtime_stats["kline_chunk"] == L
            r = rhs - P.apply(np.concatenate([P.rho(b) for b in range(batch)])).reshape(batch, -1)
            assert np.all(np.linalg.norm(r, axis=1) <= 1.001e-10 * np.linalg.norm(rhs, axis=1)), L
            its.append(max(i["iterations"] for i in info))
    assert max(its) - min(its) <= 2 + max(its) // 4, its


@pytest.mark.parametrize("n_el,nk,order,batch", [(31, 68, 3, 152), (9, 64, 1, 500)])
def test_gram_schmidt_many_problems(built_lib, n_el, nk, order, batch):
    """More problems than resident blocks: a block of the inner Arnoldi's kernels takes several pieces of a problem,
    the last one ragged.  Every problem meets the tolerance by its own FP64 residual."""
    from real_space_dg_gb300 import Problem1D
    spec, mat, E, efl, efr, m = small_rtd(n_el=n_el, nk=nk, order=order, bias=0.05)
    with Problem1D(n_el=n_el, n_local=order + 1, nk=nk, l_xi=spec.l_xi_m, batch=batch, precision="mixed",
                   inner_restart=21) as P:
        for b in range(batch):
            P.set_potential(b, mat["x"], E * (1 + 0.1 * b / batch), m, spec.m_rel, spec.temp_k, efl, efr)
        st, info = P.solve(tol=1e-10, maxit=60)
        rho = np.concatenate([P.rho(b) for b in range(batch)])
        rhs = P.rhs().reshape(batch, -1)
        r = rhs - P.apply(rho).reshape(batch, -1)
        assert st == 0
        assert np.all(np.linalg.norm(r, axis=1) <= 1.001e-10 * np.linalg.norm(rhs, axis=1))


@pytest.mark.parametrize("n_el,nk,nxi,order,batch,emulated", [
    (116, 256, 256, 3, 1, True), (153, 256, 260, 2, 2, True), (58, 512, 512, 1, 1, True), (239, 252, 256, 1, 1, True),
    (114, 256, 256, 3, 1, False), (400, 190, 190, 1, 1, False)])
def test_large_fp64_transforms(built_lib, n_el, nk, nxi, order, batch, emulated):
    """FP64 handles on both sides of 3e7 entries and nodes (and an Nk that is no multiple of 4): the operator
    against the oracle's, 1e-13 of |A x| as two FP64 sums of up to 512 terms may differ, and an Arnoldi solve whose steps
    use that the flux is inverted, by the oracle's residual."""
    from real_space_dg_gb300 import Problem1D
    spec, mat, E, efl, efr, m = small_rtd(n_el=n_el, nk=nk, order=order, n_xi=nxi, bias=0.05)
    op = krylov.Operator1D(mat, dg1d.init_params(mat, efl, efr, E, m), E)
    rng = np.random.default_rng(nk)
    with Problem1D(n_el=n_el, n_local=order + 1, nk=nk, n_xi=nxi, l_xi=spec.l_xi_m, batch=batch) as P:
        for b in range(batch):
            P.set_potential(b, mat["x"], E, m, spec.m_rel, spec.temp_k, efl, efr)
        x = rng.normal(size=(batch, P.N)) + 1j * rng.normal(size=(batch, P.N))
        P.profile(on=True, reset=True)
        y = P.apply(x).reshape(batch, -1)
        prof = P.profile(on=False, reset=True)
        assert (prof["gemm_f64_tc"][2] > 0) == emulated
        for b in range(batch):
            want = op.apply(x[b])
            assert np.linalg.norm(y[b] - want) <= 1e-13 * np.linalg.norm(want)
        st, info = P.solve(tol=1e-9, maxit=60)
        rhs = P.rhs().reshape(batch, -1)
        assert st == 0
        for b in range(batch):
            r = rhs[b] - op.apply(P.rho(b))
            assert np.linalg.norm(r) <= 1.01e-9 * np.linalg.norm(rhs[b])
