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
