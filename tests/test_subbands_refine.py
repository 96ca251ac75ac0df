"""The FP32 start and the FP64 refinement of the subband eigensolve where they hand over to each other and to
the bisection: eigenvalues of both signs and near zero, close pairs, ties of magnitude, rows and modes around the
number of lanes, entries beyond the FP32 range; against a dense symmetric eigensolve."""
import numpy as np
import pytest

from oracle import subbands as S

pytestmark = pytest.mark.gpu


def _solve(me, V, dy, nm):
    from real_space_dg_gb300.subbands import SubbandSolver
    with SubbandSolver(me.shape[0], me.shape[1], me.shape[2], nm) as s:
        return s.solve(me, V, dy)


def _check(me, V, dy, nm):
    """Eigenvalues to 16 eps of the spectral radius (a few roundings of the pivots), residuals to 64 eps of it, and
    the |lambda| of the nm smallest."""
    E, Vs = _solve(me, V, dy, nm)
    for iv in range(me.shape[0]):
        for ix in range(me.shape[1]):
            H = S.transversal_hamiltonian(me[iv, ix], V[ix], dy)
            d = np.concatenate([[1.0], np.cumprod(np.sqrt(np.diag(H, -1) / np.diag(H, 1)))])
            w, U = np.linalg.eigh(H * d[None, :] / d[:, None])
            rad = np.abs(w).max()
            want = np.sort(np.sort(np.abs(w))[:nm])
            assert np.abs(np.sort(np.abs(E[iv, ix])) - want).max() <= 16 * 2.3e-16 * rad
            assert np.all(np.diff(E[iv, ix]) >= -2e-16 * rad)
            for k in range(nm):
                v = Vs[iv, ix, k]
                assert abs(np.linalg.norm(v) - 1) < 1e-13 and v[-1] >= 0
                # in the symmetric form, so that the bound does not depend on the scaling of the end rows
                r = (H @ v - E[iv, ix, k] * v) / d
                assert np.linalg.norm(r) <= 64 * 2.3e-16 * rad * np.linalg.norm(v / d)
    return E


def _well(ny, x, dy, depth=0.0):
    y = np.arange(ny) * dy
    return np.stack([depth + 0.4 * ((y - y.mean()) / y.mean()) ** 2 * (1 + 0.05 * i) for i in range(x)])


@pytest.mark.parametrize("ny,nm", [(3, 1), (3, 3), (4, 2), (31, 5), (32, 8), (33, 11), (64, 16), (65, 17), (96, 32),
                                   (300, 3), (1024, 2)])
def test_sizes(built_lib, ny, nm):
    rng = np.random.default_rng(ny)
    me = rng.uniform(0.15, 0.6, (2, 5, ny))
    _check(me, _well(ny, 5, 0.1) + 0.02 * rng.normal(size=(5, ny)), 0.1, nm)


@pytest.mark.parametrize("shift", [-0.31, -1.0, -5.0])
def test_both_signs(built_lib, shift):
    me = np.full((1, 40, 71), 0.19)
    V = _well(71, 40, 0.1) + shift + np.linspace(0, 0.2, 40)[:, None]     # levels pass through zero
    _check(me, V, 0.1, 9)


@pytest.mark.parametrize("barrier", [0.5, 3.0, 30.0])
def test_close_pairs(built_lib, barrier):
    """Double wells: pairs from well separated to equal in FP32 and to rounding level in FP64.  Only their
    eigenvalues are compared: the vectors of a pair at rounding level are any basis of its plane."""
    ny, nm, dy = 121, 6, 0.1
    me = np.full((1, 3, ny), 0.3)
    y = np.arange(ny) * dy
    V = np.stack([np.where(np.abs(y - y.mean()) < 1.5, barrier * (1 + 0.1 * i), 0.0) for i in range(3)])
    E, _ = _solve(me, V, dy, nm)
    for ix in range(3):
        w = np.linalg.eigvalsh(S.transversal_hamiltonian(me[0, ix], V[ix], dy))
        assert np.abs(E[0, ix] - w[:nm]).max() <= 16 * 2.3e-16 * w[-1]


def test_ties(built_lib):
    """V = -2 t makes the spectrum symmetric about zero: every magnitude occurs twice."""
    ny, dy, m = 40, 0.25, 0.2
    t = S.hopping_scale(dy) / m
    for nm in (1, 3, 4):
        E, _ = _solve(np.full((1, 2, ny), m), np.full((2, ny), -2 * t), dy, nm)
        w = np.sort(np.abs(2 * t * np.cos(np.arange(1, ny + 1) * np.pi / (ny + 1))))[:nm]
        assert np.abs(np.sort(np.abs(E[0])) - w).max() <= 16 * 2.3e-16 * 4 * t


def test_beyond_fp32(built_lib):
    """Potentials and hoppings outside the FP32 range go through the bisection."""
    me = np.full((1, 3, 30), 0.3)
    V = _well(30, 3, 0.1)
    V[1, 10] = 1e40
    E, _ = _solve(me, V, 0.1, 4)
    for ix in (0, 2):
        w = np.linalg.eigvalsh(S.transversal_hamiltonian(me[0, ix], V[ix], 0.1))
        assert np.abs(E[0, ix] - w[:4]).max() <= 16 * 2.3e-16 * w[-1]
    assert np.all(np.isfinite(E))


@pytest.mark.parametrize("nm,ny", [(1, 70), (2, 71), (5, 40), (8, 133)])
def test_near_ties(built_lib, nm, ny):
    """Magnitudes of opposite sign from 1e-3 to 1e-13 of the radius apart, either one the smaller: above the rounding
    of the counts the kept set is that of the dense solve."""
    dy = 0.1
    base = _well(ny, 1, dy)[0] + 0.02 * np.random.default_rng(ny).normal(size=ny)
    me1 = np.full(ny, 0.25)
    w = np.linalg.eigvalsh(S.transversal_hamiltonian(me1, base, dy))
    rad = w[-1] - w[0]
    V, gaps = [], []
    for g in (1e-3, 3e-5, 1e-5, 1e-6, 1e-7, 1e-8, 1e-9, 1e-10, 1e-11, 1e-13):
        for s in (-1, 1):
            for j in (2, 7):
                # eigenvalues j and j + nm at -x and x + s g: the last of nm kept is one of the two
                V.append(base - 0.5 * (w[j] + w[j + nm]) + 0.5 * s * g * rad)
                gaps.append(g)
    V = np.stack(V)
    E, _ = _solve(np.tile(me1, (1, len(V), 1)), V, dy, nm)
    for ix in range(len(V)):
        u = np.linalg.eigvalsh(S.transversal_hamiltonian(me1, V[ix], dy))
        r = np.abs(u).max()
        keep = np.sort(u[np.argsort(np.abs(u))[:nm]])
        tol = 64 * 2.3e-16 * r       # numpy's eigenvalues and the device's
        if gaps[ix] * rad > 4 * tol:
            assert np.abs(np.sort(E[0, ix]) - keep).max() <= tol, (ix, gaps[ix])
        else:
            assert np.abs(np.sort(np.abs(E[0, ix])) - np.sort(np.abs(keep))).max() <= tol + gaps[ix] * rad


@pytest.mark.parametrize("ny,nm,wall", [(300, 32, 1e6), (300, 32, 1e7), (64, 4, 1e7), (300, 32, 1e12), (1024, 8, 1e8)])
def test_wall_above_the_band(built_lib, ny, nm, wall):
    """One row so far above the other levels that most or all of them lie within the counts' uncertainty around 0 (4e-6
    of the radius), up to ny candidates for 2 nm + 1 places: such slices go to the bisection.  The last row has no
    wall; both against the dense solve."""
    dy = 0.1
    V = _well(ny, 2, dy)
    V[0, ny // 3] = wall
    E, Vs = _solve(np.full((1, 2, ny), 0.3), V, dy, nm)
    for ix in range(2):
        w = np.linalg.eigvalsh(S.transversal_hamiltonian(np.full(ny, 0.3), V[ix], dy))
        want = np.sort(np.sort(np.abs(w))[:nm])
        assert np.abs(np.sort(np.abs(E[0, ix])) - want).max() <= 16 * 2.3e-16 * np.abs(w).max()
    assert np.all(np.isfinite(Vs))
