"""The reciprocal square root and reciprocal of the FP64 line-march stages against
80-bit arithmetic over all mantissas and exponents.  Their relative error is at most
1.5 x 2^-53 (the rounding of the result and half of the rounding of x y) and
1.01 x 2^-53, derived where they are defined; powers of two are exact, and the mean
of the errors is near zero."""
import ctypes

import numpy as np
import pytest

from artracfd_b200.abi import check, load_library

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _roots(x):
    lib = load_library()
    x = np.ascontiguousarray(x, dtype=np.float64)
    out = np.empty((2, x.size))
    ptr = [a.ctypes.data_as(ctypes.c_void_p) for a in (x, out[0], out[1])]
    check(lib.acfd_line_roots(*ptr, x.size), lib)
    return out


def _values(lo, hi):
    rng = np.random.default_rng(1)
    m = np.concatenate([1.0 + rng.random(1 << 20), 1.0 + np.arange(4096) / 4096.0, 2.0 - np.arange(1, 512) * 2.0 ** -52,
                        1.0 + np.arange(512) * 2.0 ** -52])
    return np.ldexp(m, rng.integers(lo, hi, m.size))


@pytest.mark.skipif(np.finfo(np.longdouble).nmant < 63, reason="needs 80-bit arithmetic on the host")
@pytest.mark.parametrize("which,lo,hi,bound", [(0, -1022, 1023, 1.5), (1, -1021, 1021, 1.01)], ids=["rsqrt", "rcp"])
def test_error_bounds(which, lo, hi, bound):
    x = _values(lo, hi)
    got = _roots(x)[which].astype(np.longdouble)
    X = x.astype(np.longdouble)
    want = 1 / (np.sqrt(X) if which == 0 else X)
    err = (got - want) / want
    assert np.abs(err).max() <= bound * U * (1 + 2.0 ** -9)  # 2^-63 of the host's own roundings
    assert abs(err.mean()) <= 0.05 * U


def test_powers_of_two_are_exact():
    e = np.arange(-1020, 1021)
    r, q = _roots(np.ldexp(1.0, e))
    assert np.array_equal(q, np.ldexp(1.0, -e))
    even = e % 2 == 0
    assert np.array_equal(r[even], np.ldexp(1.0, -(e[even] // 2)))
