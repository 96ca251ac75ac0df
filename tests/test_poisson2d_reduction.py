"""The block cyclic reduction of the 2D Poisson step around its sizes: numbers of columns with every pattern
of missing neighbours (2 to 17, powers of two and their neighbours, groups of 8 cut short), every block width (4 to 32
rows, padded and full) and fixed nodes inside the grid, against the oracle's sparse LU."""
import numpy as np
import pytest

from test_poisson2d import _solve_both, density, grid

pytestmark = pytest.mark.gpu


def _check(mat, bias, method, seed=5):
    n = density(mat, seed=seed)
    phi0 = 0.05 * np.random.default_rng(seed).normal(size=(mat["Nx"], mat["Ny"]))
    if mat.get("dg"):
        phi0[:, -1] = phi0[:, 0]
    want, err_o, io, got, err_g, ig = _solve_both(mat, n, phi0, bias, method)
    # the bar of the other Poisson tests: condition numbers up to ~1e4 times the rounding of the factorisation
    assert np.abs(got - want).max() <= 1e-11 * max(1.0, np.abs(want).max())
    assert abs(err_g - err_o) <= 1e-10 * max(1.0, err_o)
    assert ig["converged"]


@pytest.mark.parametrize("nx", [3, 4, 5, 7, 8, 9, 15, 16, 17, 24, 31, 33, 65])
def test_column_counts(built_lib, nx):
    _check(grid(nx=nx, ny=6, seed=nx), 0.3, "direct")


@pytest.mark.parametrize("ny,periodic", [(1, False), (2, False), (3, True), (4, False), (5, False), (8, False), (9, True),
                                         (12, False), (15, False), (17, True), (21, False), (25, True), (30, False),
                                         (32, False), (33, True)])
def test_block_widths(built_lib, ny, periodic):
    _check(grid(nx=19, ny=ny, seed=ny, periodic=periodic), 0.2, "newton-raphson")


@pytest.mark.parametrize("method", ["direct", "newton-raphson"])
def test_fixed_nodes_inside(built_lib, method):
    """Gates inside the grid: single nodes, a whole column, and a column next to the contact."""
    mat = grid(nx=22, ny=7, seed=3)
    b = np.zeros((22, 7), dtype=int)
    b[[0, -1], :] = 1
    b[5, 2] = b[6, 2] = b[13, 6] = 1
    b[9, :] = 1
    b[1, 1:4] = 1
    vbc = np.where(b, np.random.default_rng(1).uniform(-0.2, 0.2, (22, 7)), 0.0)
    mat.update(boundary=b, Vbc=vbc)
    _check(mat, 0.0, method)


@pytest.mark.parametrize("nx", [2, 6, 40])
def test_neumann_ends(built_lib, nx):
    _check(grid(nx=nx, ny=5, seed=nx, poisson=dict(xBoundary="neumann")), 0.0, "newton-raphson")


@pytest.mark.parametrize("batch,cfg", [(1025, dict(nx=19, ny=6)), (2050, dict(nx=9, ny=14, periodic=True)),
                                       (65_600, dict(nx=3, ny=2))])
def test_any_number_of_bias_points(built_lib, batch, cfg):
    """Batches beyond a group of launches and beyond a grid's second dimension: the points around the groups' edges
    have the bits that they have alone."""
    from real_space_dg_gb300.poisson2d import Poisson2D
    mat = grid(seed=batch, **cfg)
    nx, ny = mat["Nx"], mat["Ny"]
    rng = np.random.default_rng(batch)
    n = density(mat) * rng.uniform(0.5, 1.5, (batch, 1, 1))
    phi0 = 0.05 * rng.normal(size=(batch, nx, ny))
    if cfg.get("periodic"):
        phi0[..., -1] = phi0[..., 0]
    bias = rng.uniform(0.0, 0.4, batch)
    with Poisson2D(mat, batch=batch) as op:
        phi, dens, info = op.solve(n, phi0, bias, method="newton-raphson")
    assert all(i["converged"] for i in info)
    with Poisson2D(mat) as op:
        for b in (0, 1, 1023, 1024, batch - 1):
            p1, d1, i1 = op.solve(n[b], phi0[b], bias[b], method="newton-raphson")
            assert np.array_equal(p1, phi[b]) and np.array_equal(d1, dens[b]) and i1 == info[b]
