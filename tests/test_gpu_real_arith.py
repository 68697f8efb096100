"""The real forms of the FP64 kernels (models whose vertices are all real) and the
column-distributed pivoted QR, at sizes around their tiles, against the CPU oracle and against
the complex products of the same model (FLAG_COMPLEX_ARITH).

G at every stabilisation point within 1e-10 relative of the oracle's, the plain form's bound;
D of a decomposition within 1e-10 relative and its reconstruction within 1e-10 (the bounds of
the parity tests)."""
import numpy as np
import pytest

import oracle
from alf_gb300 import model as mdl, rng
from alf_gb300.sweep import FLAG_COMPLEX_ARITH, Chains, decompose as gpu_decompose
from parity_util import compare_record

pytestmark = pytest.mark.gpu


def _relmax(a, b):
    return np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300)


def _record(m, flags, f0, u, precision="fp64", chains=1):
    g = Chains(m, n_chains=chains, precision=precision, flags=flags)
    for c in range(chains):
        g.set_fields(c, f0)
    g.init_state()
    g.set_recording(True)
    g.sweep(np.stack([u] * chains))
    r = [g.record(c) for c in range(chains)]
    f = g.fields(chains - 1)
    g.close()
    return r, f


# N = 9 .. 225: one to sixteen columns per CTA, row counts around 8, 16, 32, 64, 128, 224
@pytest.mark.parametrize("L1,L2", [(3, 3), (4, 4), (5, 3), (3, 11), (8, 8), (5, 13), (9, 11), (15, 15)])
def test_real_sweep_matches_oracle_and_complex_products(L1, L2):
    m = mdl.hubbard("square", L1, L2, U=4.0, beta=0.8, dtau=0.1, nwrap=3)
    f0 = rng.initial_fields(5, 0, m.n_op, m.ltrot)
    u = rng.sweep_uniforms(5, 0, m.n_op, m.ltrot, 0)
    (rr,), fr = _record(m, 0, f0, u)
    (rc,), fc = _record(m, FLAG_COMPLEX_ARITH, f0, u)
    o = oracle.Oracle(m)
    o.set_fields(f0)
    o.init_state()
    o.record(1)
    o.sweep(u)
    ro = o.recorded()
    compare_record(rr, ro, u, m.n_op, m.ltrot, m.nwrap, g_tol=1e-10, relative=True, exact_sequence=True,
                   ratio_median=1e-12)
    assert np.array_equal(rr["acc"], rc["acc"]) and np.array_equal(fr, fc)
    assert _relmax(rr["G"], rc["G"]) <= 1e-10
    assert np.all(rr["G"].imag == 0.0)


# the QR's cluster sizes (1, 2, 4, 8, 16 CTAs) and its column and row remainders
@pytest.mark.parametrize("N", [1, 2, 15, 16, 17, 31, 33, 95, 97, 130, 225, 321])
@pytest.mark.parametrize("side", ["r", "l"])
def test_decompose_sizes(N, side):
    rs = np.random.default_rng(N)
    X = rs.standard_normal((N, N)) + 1j * rs.standard_normal((N, N))
    D = 10.0 ** rs.uniform(-8, 8, N)
    V = np.eye(N) + np.triu(rs.standard_normal((N, N)), 1) * (0.3 / np.sqrt(N))
    # copies: a 1 x 1 transpose is a view, and the wrappers decompose in place
    U, d, W = gpu_decompose(side, X.copy(), D.astype(complex), V.astype(complex))
    _, do, _ = oracle.decompose(side, X.copy(), D.astype(complex), V.astype(complex))
    A = (X * D) @ (V if side == "r" else V.conj().T)
    R = U @ np.diag(d) @ (W if side == "r" else W.conj().T)
    assert np.max(np.abs(d / do - 1.0)) < 1e-10
    assert _relmax(R, A) < 1e-10
    assert np.max(np.abs(U.conj().T @ U - np.eye(N))) < 1e-12


# reflectors that are the identity, and norms that tie (the first column wins): the oracle's pivots,
# so the same factors
@pytest.mark.parametrize("N", [2, 17, 40, 130])
@pytest.mark.parametrize("kind", ["identity", "permutation", "upper"])
def test_decompose_ties(N, kind):
    X = np.eye(N, dtype=complex)
    if kind == "permutation":
        X = X[np.random.default_rng(N).permutation(N)]
    if kind == "upper":  # columns of equal norm, all of whose reflectors are trivial
        X = np.triu(np.ones((N, N)), 0) / np.sqrt(np.arange(1, N + 1))[None, :] * (1.0 + 0j)
    one, V = np.ones(N, dtype=complex), np.eye(N, dtype=complex)
    U, d, W = gpu_decompose("r", X.copy(), one, V)
    Uo, do, Wo = oracle.decompose("r", X.copy(), one, V)
    assert _relmax(U @ np.diag(d) @ W, X) < 1e-12
    if kind != "upper":  # norms equal to the last bit
        assert np.max(np.abs(U - Uo)) < 1e-14 and np.max(np.abs(W - Wo)) < 1e-14


# right-hand sides per CTA (2, 4, 8), row blocks of 32 and their remainders, both solve
# directions, complex factors
@pytest.mark.parametrize("N", [1, 5, 31, 32, 33, 64, 100, 257, 320])
@pytest.mark.parametrize("nvar", [1, 2])
def test_cgr_sizes(N, nvar):
    from alf_gb300.sweep import cgr as gpu_cgr
    rs = np.random.default_rng(1000 + N)
    q = lambda: np.linalg.qr(rs.standard_normal((N, N)) + 1j * rs.standard_normal((N, N)))[0]
    UR, UL = q(), q()
    VR, VL = (np.eye(N) + np.triu(rs.standard_normal((N, N)) + 1j * rs.standard_normal((N, N)), 1) * (0.3 / np.sqrt(N))
              for _ in range(2))
    DR = np.sort(10.0 ** rs.uniform(-6, 6, N))[::-1].astype(complex)
    DL = np.sort(10.0 ** rs.uniform(-6, 6, N))[::-1].astype(complex)
    G, ph = gpu_cgr(nvar, UR.copy(), DR, VR.copy(), UL.copy(), DL, VL.copy())
    Go, pho = oracle.cgr(nvar, UR.copy(), DR, VR.copy(), UL.copy(), DL, VL.copy())
    assert _relmax(G, Go) < 1e-10
    assert abs(ph - pho) < 1e-10


# batched real solves and Q columns (eight vectors per CTA, one warp per column), and TAU_M's 2N
# system, against the complex products: the quartets within 1e-10 of their largest entry
@pytest.mark.parametrize("chains,L1,L2", [(1, 4, 3), (6, 7, 5), (9, 9, 8)])
def test_real_tau_matches_complex_products(chains, L1, L2):
    m = mdl.hubbard("square", L1, L2, U=4.0, beta=0.8, dtau=0.1, nwrap=3)
    u = np.stack([rng.sweep_uniforms(7, c, m.n_op, m.ltrot, 0) for c in range(chains)])
    out = []
    for flags in (0, FLAG_COMPLEX_ARITH):
        g = Chains(m, n_chains=chains, ltau=1, flags=flags)
        for c in range(chains):
            g.set_fields(c, rng.initial_fields(7, c, m.n_op, m.ltrot))
        g.init_state()
        _, tau = g.sweep(u, measure=True, keep=lambda k, c, nt: k == 1 and c in (0, chains - 1))
        out.append((tau, [g.fields(c) for c in range(chains)]))
        g.close()
    (ta, fa), (tb, fb) = out
    assert all(np.array_equal(x, y) for x, y in zip(fa, fb)) and len(ta) == len(tb) > 0
    for (c, nt, qa, _), (c2, nt2, qb, _) in zip(ta, tb):
        assert (c, nt) == (c2, nt2)
        for a, b in zip(qa, qb):
            assert _relmax(a, b) <= 1e-10


# the delayed-update block: 2 .. 32 positions, few and nearly all of them accepted (one and two
# columns of Y per warp in the flush operands), one and several blocks per slice; plain and mixed
# form, real and complex arithmetic.  Plain form: the oracle's accept sequence and G; mixed form on
# complex arithmetic runs its visits in double-float: 1e-5, the bound of its parity tests.
@pytest.mark.parametrize("delay", [2, 7, 17, 32])
@pytest.mark.parametrize("U", [0.2, 4.0])
def test_update_blocks(delay, U):
    m = mdl.hubbard("square", 6, 6, U=U, beta=0.8, dtau=0.1, nwrap=4)
    f0 = rng.initial_fields(9, 0, m.n_op, m.ltrot)
    u = rng.sweep_uniforms(9, 0, m.n_op, m.ltrot, 0)
    o = oracle.Oracle(m)
    o.set_fields(f0)
    o.init_state()
    o.record(1)
    o.sweep(u)
    ro = o.recorded()
    for precision, flags, tol in (("fp64", 0, 1e-10), ("fp64", FLAG_COMPLEX_ARITH, 1e-10), ("mixed", 0, 1e-10),
                                  ("mixed", FLAG_COMPLEX_ARITH, 1e-5)):
        g = Chains(m, precision=precision, flags=flags, delay_k=delay)
        g.set_fields(0, f0)
        g.init_state()
        g.set_recording(True)
        g.sweep(u[None])
        rg = g.record(0)
        g.close()
        compare_record(rg, ro, u, m.n_op, m.ltrot, m.nwrap, g_tol=tol, relative=True,
                       exact_sequence=precision == "fp64")


# the real FP64 products: 16 x 16 tiles with one, two and four slices of K (few and many tiles, K
# remainders of 4 and 64), 64 x 64 tiles (24 chains), every operand form of the sweep with its
# permutations, triangles and scales: against the complex products, 1e-10 relative
@pytest.mark.parametrize("chains,L1,L2", [(1, 2, 3), (2, 5, 5), (5, 8, 8), (3, 11, 7), (24, 13, 10)])
def test_real_products(chains, L1, L2):
    m = mdl.hubbard("square", L1, L2, U=4.0, beta=0.6, dtau=0.1, nwrap=2)
    u = np.stack([rng.sweep_uniforms(11, c, m.n_op, m.ltrot, 0) for c in range(chains)])
    out = []
    for flags in (0, FLAG_COMPLEX_ARITH):
        g = Chains(m, n_chains=chains, flags=flags)
        for c in range(chains):
            g.set_fields(c, rng.initial_fields(11, c, m.n_op, m.ltrot))
        g.init_state()
        g.sweep(u)
        out.append(([g.green(c) for c in range(chains)], [g.fields(c) for c in range(chains)], g.phase()))
        g.close()
    (ga, fa, pa), (gb, fb, pb) = out
    assert all(np.array_equal(x, y) for x, y in zip(fa, fb))
    assert all(_relmax(x, y) <= 1e-10 for x, y in zip(ga, gb))
    assert np.max(np.abs(pa - pb)) <= 1e-10


# the tensor-core products of the FP64 form (62-bit digits): forced on (FLAG_TENSOR_WIDE) against the
# FP64 pipes (FLAG_NO_TENSOR_GEMM), real and complex, N around the digit widths' and tiles' edges
# (16, 32, 64, 128), one and several matrices per launch; accept sequences equal, G to 1e-10
@pytest.mark.parametrize("chains,L1,L2", [(1, 3, 5), (3, 8, 8), (2, 5, 13), (1, 8, 16), (2, 3, 43)])
@pytest.mark.parametrize("flags", [0, FLAG_COMPLEX_ARITH])
def test_fp64_tensor_products(chains, L1, L2, flags):
    from alf_gb300.sweep import FLAG_NO_TENSOR_GEMM, FLAG_TENSOR_WIDE
    m = mdl.hubbard("square", L1, L2, U=4.0, beta=0.4, dtau=0.1, nwrap=2)
    u = np.stack([rng.sweep_uniforms(13, c, m.n_op, m.ltrot, 0) for c in range(chains)])
    out = []
    for fl in (FLAG_TENSOR_WIDE, FLAG_NO_TENSOR_GEMM):
        g = Chains(m, n_chains=chains, flags=fl | flags, ltau=1)
        for c in range(chains):
            g.set_fields(c, rng.initial_fields(13, c, m.n_op, m.ltrot))
        g.init_state()
        g.set_recording(True)
        _, tau = g.sweep(u, measure=True, keep=lambda k, c, nt: k == 1)
        out.append(([g.record(c) for c in range(chains)], tau))
        g.close()
    for a, b in zip(out[0][0], out[1][0]):
        assert np.array_equal(a["acc"], b["acc"])
        assert _relmax(a["G"], b["G"]) <= 1e-10
    for (c, nt, qa, _), (_, _, qb, _) in zip(out[0][1], out[1][1]):
        assert all(_relmax(x, y) <= 1e-10 for x, y in zip(qa, qb))


# the complex FP64 products of a model with complex vertices: one and two slices of K, few and many
# tiles, remainders of 16 and 32: against the oracle
@pytest.mark.parametrize("chains,L1,L2", [(1, 1, 3), (1, 3, 3), (2, 5, 3), (6, 5, 4), (114, 8, 8)])
def test_complex_products(chains, L1, L2):
    from alf_gb300.sweep import FLAG_NO_TENSOR_GEMM
    m = mdl.kondo(L1, L2, JK=1.5, Uf=2.0, beta=0.4, dtau=0.1, nwrap=2)
    f0 = rng.initial_fields(15, 0, m.n_op, m.ltrot)
    u = rng.sweep_uniforms(15, 0, m.n_op, m.ltrot, 0)
    r, _ = _record(m, FLAG_NO_TENSOR_GEMM, f0, u, chains=chains)
    o = oracle.Oracle(m)
    o.set_fields(f0)
    o.init_state()
    o.record(1)
    o.sweep(u)
    ro = o.recorded()
    for k in (0, chains - 1):
        compare_record(r[k], ro, u, m.n_op, m.ltrot, m.nwrap, g_tol=1e-10, relative=True, exact_sequence=True)


# Q over all panels in one launch: 9 and 13 row blocks per column (12 and 24 held by a lane), one and
# several columns per warp, an explicit Q and CGR2_2's application to general columns; against the complex products
@pytest.mark.parametrize("chains,L1,L2", [(1, 13, 10), (1, 20, 10), (6, 13, 10)])
def test_real_q_of_large_systems(chains, L1, L2):
    test_real_tau_matches_complex_products(chains, L1, L2)


# checkerboard bonds, all families and the scalings in one launch: one and eight columns (rows) per CTA
# (1 and 24 chains), remainders, real and complex arithmetic: against the oracle
@pytest.mark.parametrize("flags", [0, FLAG_COMPLEX_ARITH])
@pytest.mark.parametrize("lattice,chains,L1,L2", [("square", 1, 4, 2), ("square", 24, 6, 6), ("honeycomb", 2, 3, 3),
                                                  ("honeycomb", 24, 4, 3)])
def test_bond_launches(lattice, chains, L1, L2, flags):
    m = mdl.hubbard(lattice, L1, L2, U=4.0, chem=0.2, beta=0.6, dtau=0.1, nwrap=3, checkerboard=True)
    f0 = rng.initial_fields(17, 0, m.n_op, m.ltrot)
    u = rng.sweep_uniforms(17, 0, m.n_op, m.ltrot, 0)
    r, _ = _record(m, flags, f0, u, chains=chains)
    o = oracle.Oracle(m)
    o.set_fields(f0)
    o.init_state()
    o.record(1)
    o.sweep(u)
    ro = o.recorded()
    for k in (0, chains - 1):
        compare_record(r[k], ro, u, m.n_op, m.ltrot, m.nwrap, g_tol=1e-10, relative=True, exact_sequence=True)
