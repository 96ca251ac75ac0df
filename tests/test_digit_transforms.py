"""The FP64 transforms as digit products on the tensor cores: non-finite inputs, the choice between them and the native
kernels, and what they do where memory or the grid is short."""
import numpy as np
import pytest

from conftest import small_rtd

pytestmark = pytest.mark.gpu


def _problem(n_el, nk, nxi, order, batch=1, **kw):
    from real_space_dg_gb300 import Problem1D
    spec, mat, E, efl, efr, m = small_rtd(n_el=n_el, nk=nk, order=order, n_xi=nxi)
    P = Problem1D(n_el=n_el, n_local=order + 1, nk=nk, n_xi=nxi, l_xi=spec.l_xi_m, batch=batch, **kw)
    for b in range(batch):
        P.set_potential(b, mat["x"], E * (1 + 0.1 * b), m, spec.m_rel, spec.temp_k, efl, efr)
    return P


@pytest.mark.parametrize("kind", [dict(fp64_tc=True), dict(precision="mixed")])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, complex(0.0, np.nan)])
@pytest.mark.parametrize("n_el,nk,nxi,order,at", [(4, 32, 32, 1, 0), (5, 64, 72, 2, 40), (3, 260, 512, 1, 259)])
def test_non_finite_inputs(built_lib, n_el, nk, nxi, order, at, value, kind):
    """One infinity or NaN at wave number `at` of one node of the middle element: the operator is non-finite exactly where
    it is with the native kernels (NaN where a NaN makes it so), and the rest agrees (1e-12 of |A x|, as without it)."""
    out = []
    for kw in (dict(), kind):
        with _problem(n_el, nk, nxi, order, **kw) as P:
            rng = np.random.default_rng(nk)
            x = rng.normal(size=P.N) + 1j * rng.normal(size=P.N)
            x[(n_el // 2 * (order + 1) + 1) * nk + at] = value
            out.append(P.apply(x))
    want, got = out
    finite = np.isfinite(want)
    assert 0 < finite.sum() < want.size
    assert np.array_equal(np.isfinite(got), finite)
    if np.isnan(value):
        assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.linalg.norm(got[finite] - want[finite]) <= 1e-12 * np.linalg.norm(want[finite])


@pytest.mark.parametrize("kind", [dict(fp64TensorCores=True), dict(precision="mixed")])
@pytest.mark.parametrize("method", ["rk4", "cn"])
def test_timeouts_reach_the_transient(built_lib, kind, method):
    """A wait of the products that ran out (its flag raised from the host; no kernel runs with it) ends a transient and
    a timing run with an error, as it does a solve: the state after it is not the integrated one."""
    from real_space_dg_gb300 import WignerError, _lib, devices
    from real_space_dg_gb300.rtd import RTDSweep
    mat = small_rtd(n_el=10, nk=32, order=2)[1]
    S = RTDSweep(dict(mat, dy_norm_nm=devices.density_normalisation_nm(mat)), 1, dict(transportMaxCycles=60, **kind))
    try:
        S.set(0, 0.05)
        assert S.run()[0] == 0
        assert S.transient(1e-17, 2, method)[0] == 0 and S.P.apply_time("fp64", 1) > 0
        assert S.lib.wg_debug_mark_timeout(S.P.h) == _lib.WG_OK
        for call in (lambda: S.transient(1e-17, 0, method), lambda: S.P.apply_time("fp64", 1)):
            with pytest.raises(WignerError) as e:
                call()
            assert e.value.status == _lib.WG_ERR_TIMEOUT
    finally:
        S.close()


@pytest.mark.parametrize("fp64_tc,emulated", [(False, True), (True, True), (-1, False)])
def test_the_caller_chooses(built_lib, fp64_tc, emulated):
    """Above 3e7 entries and nodes the default takes the digit products; both kinds can be asked for, here and in the
    options of a sweep."""
    from real_space_dg_gb300 import devices
    from real_space_dg_gb300.rtd import RTDSweep
    with _problem(58, 512, 512, 3, fp64_tc=fp64_tc) as P:
        P.profile(on=True, reset=True)
        P.apply(np.ones(P.N))
        prof = P.profile(on=False, reset=True)
        assert (prof["gemm_f64_tc"][2] > 0) == emulated and (prof["gemm_f64"][2] == 0) == emulated
    mat = small_rtd(n_el=58, nk=512, order=3, n_xi=512)[1]
    S = RTDSweep(dict(mat, dy_norm_nm=devices.density_normalisation_nm(mat)), 1, dict(fp64TensorCores=fp64_tc))
    try:
        S.set(0, 0.0)
        S.P.profile(on=True, reset=True)
        S.P.apply(np.ones(S.P.N))
        assert (S.P.profile(on=False, reset=True)["gemm_f64_tc"][2] > 0) == emulated
    finally:
        S.close()


def _bytes(budget, **shape):
    import ctypes as C
    from real_space_dg_gb300 import _lib
    prm = _lib.WgParams(shape["n_el"], shape["order"] + 1, shape["nk"], shape["nxi"], 30e-9, 0.0, 1.0, _lib.WG_PREC_FP64,
                        20, budget)
    out = C.c_double()
    assert _lib.load().wg_problem_bytes(C.byref(prm), shape["batch"], C.byref(out)) == _lib.WG_OK
    return out.value


@pytest.mark.parametrize("n_el,nk,nxi,order,batch", [(116, 256, 256, 3, 1), (153, 256, 260, 2, 2), (59, 508, 512, 3, 1),
                                                     (2000, 60, 132, 1, 1)])
def test_results_do_not_depend_on_memory_or_batch(built_lib, n_el, nk, nxi, order, batch):
    """The same bits with a buffer for all digits, with an admission budget that leaves no room for one (the digits then
    take two or three passes, the last one overlapping) and alone in a batch; the estimate
    counts the buffer."""
    shape = dict(n_el=n_el, nk=nk, nxi=nxi, order=order, batch=batch)
    full, least = _bytes(0.0, **shape), _bytes(1.0, **shape)
    assert least < full
    rng = np.random.default_rng(nk)
    out, held = [], []
    for budget in (0.0, least):
        with _problem(**shape, mem_budget_bytes=budget, restart=20) as P:
            if not out:
                x = rng.normal(size=P.N * batch) + 1j * rng.normal(size=P.N * batch)
            P.profile(on=True, reset=True)
            out.append(P.apply(x))
            assert P.profile(on=False, reset=True)["gemm_f64_tc"][2] > 0
            held.append(P.device_bytes)
    assert held[0] - held[1] == full - least
    assert np.array_equal(out[0], out[1])
    with _problem(n_el, nk, nxi, order, restart=20) as P:      # problem 0 of the batch has the unscaled potential
        assert np.array_equal(P.apply(x[:P.N]), out[0][:P.N])
        P.set_rhs(0, x[:P.N])
        st, info = P.solve(tol=1e-3, maxit=1)
    with _problem(n_el, nk, nxi, order, restart=20, mem_budget_bytes=_bytes(1.0, **dict(shape, batch=1))) as P:
        P.set_rhs(0, x[:P.N])
        assert P.solve(tol=1e-3, maxit=1)[1][0]["iterations"] == info[0]["iterations"]


def test_served_without_room_for_the_digits(built_lib):
    """A server whose budget holds one slot of a large FP64 shape without the digits' buffer, and not with it."""
    from real_space_dg_gb300 import devices
    from real_space_dg_gb300.serve import Server
    spec, mat, *_ = small_rtd(n_el=58, nk=512, order=3, n_xi=512)
    mat = dict(mat, dy_norm_nm=devices.density_normalisation_nm(mat))
    least, full = (_bytes(b, n_el=58, nk=512, nxi=512, order=3, batch=1) for b in (1.0, 0.0))
    with Server(dict(precision="fp64", restart=20, maxIterations=2, transportTolerance=1e-6),
                mem_budget_bytes=0.5 * (least + full), max_slots=2) as S:
        r = S.wait(S.submit(mat, 0.0), timeout=60)
        assert r["state"] == "done" and np.all(np.isfinite(r["n"])), r["error"]
        assert least <= S.stats()["device_bytes_peak"] <= 0.5 * (least + full)


@pytest.mark.parametrize("kind", [dict(fp64_tc=True), dict(precision="mixed", inner_restart=2)])
def test_more_nodes_than_grid_rows(built_lib, kind):
    """2,098,800 nodes, more than 65,535 tiles of 32: the last problem of the handle against the same problem alone."""
    n_el, nk, order, batch = 990, 32 if "precision" in kind else 8, 3, 530
    from real_space_dg_gb300 import Problem1D
    spec, mat, E, efl, efr, m = small_rtd(n_el=n_el, nk=nk, order=order)
    rng = np.random.default_rng(0)
    out = []
    for b in (batch, 1):
        with Problem1D(n_el=n_el, n_local=order + 1, nk=nk, l_xi=spec.l_xi_m, batch=b, restart=2, **kind) as P:
            P.set_potential(b - 1, mat["x"], E, m, spec.m_rel, spec.temp_k, efl, efr)
            x = np.zeros((b, P.N), dtype=complex)
            x[-1] = rng.normal(size=P.N) + 1j * rng.normal(size=P.N) if not out else out[0][0]
            out.append((x[-1].copy(), P.apply(x).reshape(b, -1)[-1].copy()))
    assert np.array_equal(out[0][1], out[1][1]) and np.linalg.norm(out[1][1]) > 0


@pytest.mark.parametrize("kind", ["normal", "decades in k", "decades over elements"])
@pytest.mark.parametrize("n_el,nk,nxi,order", [(6, 16, 16, 1), (4, 36, 52, 2), (5, 64, 64, 3), (40, 60, 64, 1)])
def test_all_digits_count(built_lib, n_el, nk, nxi, order, kind):
    """The potential term (the flux is made negligible by a heavy m_diff) against the native kernels, per element.  Native
    sums of up to 32 pairs carry about sqrt(32) / 2 roundings, 3e-16 a transform, the digits one, so both transforms
    differ by about 5e-16 of the result: 8e-16 is allowed.  The largest entry of a column in units of its rms is about 3,
    so seven digits of 7 bits (2^-50 of it per entry) are off by 1.5e-15 a transform at least (1.8e-14 measured)."""
    rng = np.random.default_rng(nk)
    out = []
    for tc in (-1, True):
        with _problem(n_el, nk, nxi, order, fp64_tc=tc, m_diff=1e-22) as P:
            if not out:
                x = rng.normal(size=(n_el, order + 1, nk)) + 1j * rng.normal(size=(n_el, order + 1, nk))
                if kind == "decades in k":
                    x *= 10.0 ** rng.uniform(-12, 0, (1, 1, nk))
                if kind == "decades over elements":
                    x *= 10.0 ** rng.uniform(-100, 100, (n_el, 1, 1))
                    x[1::2] = 0.0     # the flux takes one node of a neighbour
            out.append(P.apply(x.ravel()).reshape(n_el, -1))
    want, got = out
    on = np.linalg.norm(want, axis=1) > 0 if kind != "decades over elements" else np.arange(n_el) % 2 == 0
    assert np.all(np.linalg.norm((got - want)[on], axis=1) <= 8e-16 * np.linalg.norm(want[on], axis=1))
