"""The reciprocal of the subband and Poisson pivots against the correctly rounded 1 / x."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rcp(x):
    from real_space_dg_gb300 import _lib
    x = np.ascontiguousarray(x, dtype=float)
    y = np.empty_like(x)
    assert _lib.load().wg_debug_rcp(_lib.dptr(x), _lib.dptr(y), x.size) == _lib.WG_OK
    return y


def test_one_unit_of_the_last_place(built_lib):
    """|y - 1/x| <= 0.5 + 2^-3 units (one rounding and e^3 < 2^-56): one unit from the rounded quotient at most, over all
    exponents whose reciprocal is normal, with the mantissas around powers of two and where the instruction's 20 bits end."""
    rng = np.random.default_rng(0)
    e = np.arange(-1022, 1022)
    frac = [1.0, np.nextafter(1.0, 2.0), np.nextafter(2.0, 1.0), 1.5, 4.0 / 3, 1 + 2.0 ** -20, 1 + 2.0 ** -20 - 2.0 ** -52,
            1 + 2.0 ** -21, 2 - 2.0 ** -20] + list(rng.uniform(1, 2, 300))
    x = np.ldexp(np.array(frac)[:, None], e[None, :]).ravel()
    x = np.concatenate([x, -x])
    want = 1.0 / x
    assert np.all(np.abs(_rcp(x) - want) <= np.spacing(np.abs(want)))


def test_beyond_its_range(built_lib):
    x = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -2.0 ** -1023, 2.0 ** -1030])
    assert np.all(np.isnan(_rcp(x)))
    assert np.array_equal(_rcp(np.array([2.0 ** 1022, -2.0 ** 1023, 1.7976931348623157e308])), [2.0 ** -1022, 0.0, 0.0])
