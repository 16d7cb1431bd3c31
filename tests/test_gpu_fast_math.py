"""The quotients and roots that carry fast mode (div_nr, rsqrt_products) against
80-bit values, over operands from 2^-60 to 2^60.

Bounds, in units u = 2^-53 of relative error, from the operations: the quotient takes
the rounding of a*y and the last one (2 u), and the third power of the seed's error
(2^-19.9) is 0.01 u; in the products of the root the rounding of x*y enters by half
through the residual, beside the product's own and the last one (a/sqrt(b): 2.5 u,
sqrt(b): 1.5 u), and a seed within 2^-20 leaves 0.02 u."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def _operands(n):
    rng = np.random.default_rng(7)
    a = np.exp2(rng.uniform(-60, 60, n)) * rng.choice([-1.0, 1.0], n)
    b = np.exp2(rng.uniform(-60, 60, n))
    # significands at the ends of a binade, and equal operands
    ends = np.array([1.0, 1.0 + 2 ** -52, 2.0 - 2 ** -52, 4.0 - 2 ** -51, 1.5, 3.0])
    b[:6 * 121] = (ends[:, None] * np.exp2(np.arange(-60, 61))[None, :]).ravel()
    a[6 * 121:1000] = b[6 * 121:1000]
    return a, b


def test_fast_quotients_and_roots_within_their_bounds():
    from gaukuk_b200 import _lib
    n = 1 << 20
    a, b = _operands(n)
    out = np.empty((3, n))
    dp = ctypes.POINTER(ctypes.c_double)
    _lib.check(_lib.load().gk_fastmath_eval(n, a.ctypes.data_as(dp), b.ctypes.data_as(dp),
                                            out.ctypes.data_as(dp)))
    al, bl = a.astype(np.longdouble), b.astype(np.longdouble)
    for got, ref, bound in zip(out, (al / bl, al / np.sqrt(bl), np.sqrt(bl)), (2.02, 2.55, 1.55)):
        assert float(np.max(np.abs(got / ref - 1))) <= bound * U
