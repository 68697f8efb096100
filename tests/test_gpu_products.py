"""The digit-sliced tensor-core products: what an output depends on, and how far it is off."""
import os

import numpy as np
import pytest

from alf_gb300 import _lib, build, model as mdl, rng
from alf_gb300.sweep import FLAG_TENSOR_WIDE, Chains

pytestmark = pytest.mark.gpu


# The diagonals are combined exactly and rounded once, so an output is a function of its row and column
# alone: the same bits on the narrow tiles of one chain's grid and on the wide ones of batched grids
# (mixed form, real model: every product of the initial state on the tensor cores).  N around K = 16,
# 64, 128, where digit width and chunk count change.
@pytest.mark.parametrize("L1,L2", [(3, 4), (4, 4), (8, 8), (5, 13), (8, 16), (3, 43)])
def test_products_do_not_depend_on_the_tiles(L1, L2):
    m = mdl.hubbard("square", L1, L2, U=4.0, beta=2.0, dtau=0.1, nwrap=5)
    G = []
    for flags in (0, FLAG_TENSOR_WIDE):
        g = Chains(m, precision="mixed", flags=flags)
        g.set_fields(0, rng.initial_fields(19, 0, m.n_op, m.ltrot))
        g.init_state()
        G.append(g.green(0))
        g.close()
    assert np.all(np.isfinite(G[0])) and np.array_equal(G[0], G[1])


# ---------------------------------------------------------------------------------------------
# the FP64 form's digits by themselves: alfgpu_oz_dgemm of a library built for their 62 bits
# ---------------------------------------------------------------------------------------------
@pytest.fixture(scope="module")
def product62():
    from device import load
    L = load("oz62", os.path.join(build.CSRC, "alfgpu.cu"), ("-DOZ_TARGET_BITS=61", "-Xptxas", "-O1"))
    L.alfgpu_oz_dgemm.argtypes, L.alfgpu_oz_dgemm.restype = _lib.lib().alfgpu_oz_dgemm.argtypes, int

    def product(A, B):
        A, B = np.asfortranarray(A, dtype=np.float64), np.asfortranarray(B, dtype=np.float64)
        (m, k), n = A.shape, B.shape[1]
        C = np.zeros((m, n), order="F")
        rc = L.alfgpu_oz_dgemm(m, n, k, A.ctypes.data, m, B.ctypes.data, k, C.ctypes.data, m, 0)
        assert rc == 0, rc
        return C
    return product


def _factors(kind, m, n, k):
    r = np.random.default_rng(1000 * k + len(kind))
    if kind == "wide":  # rows and columns over 2^-40 .. 1, their largest entries at different k
        return (r.standard_normal((m, k)) * 2.0 ** r.uniform(-40, 0, (m, k)),
                r.standard_normal((k, n)) * 2.0 ** r.uniform(-40, 0, (k, n)))
    A, B = r.standard_normal((m, k)), r.standard_normal((k, n))
    if kind == "cancel" and k > 1:  # the sum cancels to 2^-60: what the digits leave is all of the error
        h = k // 2
        A[:, h:2 * h], B[h:2 * h] = A[:, :h], -B[:h]
        if k % 2:
            A[:, -1] *= 2.0 ** -60
    return A, B


# Rounding of the operands 2^-62 of the row's and column's largest entries (scales within a factor of two of
# them), dropped diagonals 7 K 4^6 2^-84 of the scales, four times that of the largest entries, with the further ones
# 1 % more, and one rounding of the result.  A plain FP64 product errs by up to 2^-53 sum_k |A_ik| |B_kj|
# a step, which is larger against the largest entries, and smaller where the largest entries of a row and a
# column do not meet: the bound and the gain are normwise.
@pytest.mark.parametrize("k", [1, 16, 17, 64, 65, 256, 448])
@pytest.mark.parametrize("kind", ["normal", "cancel", "wide"])
def test_products_of_62_bits(product62, kind, k):
    A, B = _factors(kind, 130, 70, k)
    C, F = product62(A, B), A @ B
    E = A.astype(np.longdouble) @ B.astype(np.longdouble)
    aA, aB = np.abs(A), np.abs(B)
    mA, mB = aA.max(1)[:, None], aB.max(0)[None, :]
    cut = 2.0 ** -62 * (mA * aB.sum(0)[None, :] + aA.sum(1)[:, None] * mB) + 7.07 * k * 2.0 ** -68 * mA * mB
    err, plain = (np.abs(X.astype(np.longdouble) - E).astype(np.float64) for X in (C, F))
    print(f"K = {k} {kind}: of the largest entries 2^{np.log2((err / (mA * mB)).max() + 1e-300):.1f}, plain FP64 "
          f"2^{np.log2((plain / (mA * mB)).max() + 1e-300):.1f}; of sum |A||B| 2^"
          f"{np.log2((err / (aA @ aB)).max() + 1e-300):.1f}, plain 2^{np.log2((plain / (aA @ aB)).max() + 1e-300):.1f}")
    assert np.all(err <= cut + 2.0 ** -53 * np.abs(E).astype(np.float64))
    # never worse than the plain product by more than the cut (both round the result once)
    assert (err / (mA * mB)).max() <= (plain / (mA * mB)).max() + (cut / (mA * mB)).max()


# every digit at its end (-64) in both operands: the diagonals' sums reach 9 K 4096, at K = 448 2 % below
# 2^24, where FP32 ends being exact
@pytest.mark.parametrize("k", [64, 448])
def test_products_of_extreme_digits(product62, k):
    x = -sum(64.0 * 128.0 ** -i for i in range(7))
    C = product62(np.full((130, k), x), np.full((k, 40), x))
    want = np.longdouble(x) * np.longdouble(x) * k
    assert float(abs(C.astype(np.longdouble) - want).max()) <= 0.501 * np.spacing(float(want))


def test_products_of_62_bits_end_at_448(product62):
    with pytest.raises(AssertionError, match="105"):
        product62(np.ones((8, 449)), np.ones((449, 8)))
