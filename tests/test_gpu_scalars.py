"""The scalar device functions under the sweep's kernels, by themselves."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    from device import load
    return load("scalars")


def _p(a):
    return ctypes.c_void_p(a.ctypes.data)


# FP64 -> double-float: h the nearest float, l the rest rounded once, so 2^-49 relative and the same words as
# h = float(x), l = float(x - h) (but for ties of h, where h + l is exact either way); and the way back.
# Binades from below to above the range of the bit moves, mantissas around the rounding's carries.
@pytest.mark.parametrize("lo,hi", [(-100, -69), (-71, -60), (-1, 1), (90, 102), (101, 120)])
def test_df_make(dev, lo, hi):
    r = np.random.default_rng(lo + 200)
    m = 1.0 + np.concatenate([r.random(20000), np.arange(64) * 2.0 ** -29, 1.0 - np.arange(1, 64) * 2.0 ** -30,
                              1.0 - np.arange(1, 64) * 2.0 ** -52, [0.0, 2.0 ** -24, 2.0 ** -52]])
    x = np.concatenate([np.ldexp(m, e) for e in range(lo, hi)])
    x = np.concatenate([x, -x, [0.0, -0.0]])
    h, l, back = np.empty(len(x), np.float32), np.empty(len(x), np.float32), np.empty(len(x))
    assert dev.chk_df_make(_p(x), _p(h), _p(l), _p(back), len(x)) == 0
    s = h.astype(np.float64) + l.astype(np.float64)  # exact: 24 + 24 bits with a gap of at most 4
    assert np.all(np.abs(x - s) <= 2.0 ** -49 * np.abs(x))
    hn = x.astype(np.float32)
    tie = np.abs(x - hn) * 2 == np.spacing(np.abs(hn))
    ln = (x - hn.astype(np.float64)).astype(np.float32)
    assert np.array_equal(h[~tie], hn[~tie]) and np.array_equal(l[~tie], ln[~tie])
    assert np.array_equal(back, s)


def _roots(dev, x):
    out = np.empty((5, len(x)))
    assert dev.chk_roots(_p(np.ascontiguousarray(x)), _p(out), len(x)) == 0
    return out


def _ulps(a, exact):
    """|a - exact| in units in the last place of the rounded exact value."""
    return float(np.max(np.abs(a.astype(np.longdouble) - exact) / np.spacing(np.abs(exact).astype(np.float64))))


# Every upper word of the mantissa, both exponent parities, the lower word at its ends: the approximation
# within 2^-19, so the reciprocal within half an ulp for its rounding and e^3 / 2^-53 = 1/16 at most; the
# root's Newton step leaves the rounding and the square of a few ulp.  Exact values in extended precision
# (64 or 113 bits: 2^-11 ulp or less).
@pytest.mark.parametrize("low", [0, 1, 0x80000000, 0xffffffff])
@pytest.mark.parametrize("e", [0, 1])
def test_reciprocal_and_root_all_mantissas(dev, e, low):
    hi = np.arange(1 << 20, dtype=np.uint64)
    x = (((1023 + e) << 52) | (hi << 32) | low).astype(np.uint64).view(np.float64)
    o = _roots(dev, x)
    xl = x.astype(np.longdouble)
    seed = float(np.max(np.abs(1 - xl * o[0])))
    u, v = _ulps(o[1], 1 / xl), _ulps(o[3], np.sqrt(xl))
    print(f"e = {e}, low = {low:#x}: approximation 2^{np.log2(seed):.2f}, reciprocal {u:.4f} ulp (CUDA's "
          f"{_ulps(o[2], 1 / xl):.4f}), root {v:.4f} ({_ulps(o[4], np.sqrt(xl)):.4f})")
    assert seed <= 2.0 ** -19 and u <= 0.57 and v <= 0.51


# the whole range of the corrected forms, its edges from both sides, signs; beyond it the reciprocal is CUDA's
@pytest.mark.parametrize("lo,hi", [(-900, -890), (-899, 899), (890, 900)])
def test_reciprocal_and_root_range(dev, lo, hi):
    r = np.random.default_rng(hi + 1000)
    x = np.ldexp(1.0 + r.random(200000), r.integers(lo, hi, 200000))
    x = np.concatenate([x, np.ldexp([1.0, 1.0 + 2.0 ** -52, 2.0 - 2.0 ** -52], lo), np.ldexp([1.0, 2.0 - 2.0 ** -52], hi - 1)])
    o, n = _roots(dev, np.concatenate([x, -x])), len(x)
    xl = x.astype(np.longdouble)
    assert _ulps(o[1, :n], 1 / xl) <= 0.57 and np.array_equal(o[1, n:], -o[1, :n])
    assert _ulps(o[3, :n], np.sqrt(xl)) <= 0.51


def test_reciprocal_outside(dev):
    x = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 2.0 ** -1022, 2.0 ** -1000, -2.0 ** 1000, 1.7e308])
    with np.errstate(divide="ignore", over="ignore"):
        assert np.array_equal(_roots(dev, x)[1], 1.0 / x, equal_nan=True)
