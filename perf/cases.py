"""Workloads of the sweep library, as a program that drives it meets them.

A case names a model (lattice, size, couplings, beta, dtau, Nwrap), a form ("fp64" or "mixed"), a
number of chains and what is done with them:

  sweep   one sequential sweep of every chain of one handle (``Chains.sweep``), then the state a
          driver reads back: G, the fields and the phase of every chain.  Options: the draws come
          from the caller's array ("host") or the device stream; checkerboard hopping; time-displaced
          Green functions after the sweep (ltau); scalar and lattice observables accumulated on the
          device (measure).
  many    one sweep of several handles of different sizes (``sweep_many``): the batched workload,
          one handle per lattice size.
  cgr, decompose
          the one-shot stabilisation calls on host factors.

``exact`` restates a case in plain NumPy in 64 bits: the sweep with explicit rank-1 updates and a
Green function rebuilt from the fields, the pivoted QR column by column, the assembled inverse.
"""
import math
from functools import lru_cache

import numpy as np

from alf_gb300 import lattice_obs, model, rng
from alf_gb300.sweep import Chains, cgr, decompose, sweep_many


# ------------------------------------------------------------------------------------------------
# The cases
# ------------------------------------------------------------------------------------------------
def _sweep(name, lattice, L, beta, dtau, nwrap, U, chains, form, draws="device", checkerboard=False, ltau=0,
           measure=False):
    return {"name": name, "do": "sweep", "lattice": lattice, "L1": L, "L2": L, "beta": beta, "dtau": dtau,
            "nwrap": nwrap, "U": U, "chains": chains, "form": form, "draws": draws, "checkerboard": checkerboard,
            "ltau": ltau, "measure": measure}


def listed():
    return [
        # the smallest run: a first test system, one walker, plain form (launch latency counts)
        _sweep("square4_fp64", "square", 4, 4.0, 0.1, 10, 4.0, 1, "fp64"),
        # a driver that passes its own random numbers, checkerboard hopping, a few walkers
        _sweep("square6_checkerboard", "square", 6, 4.0, 0.1, 10, 4.0, 4, "fp64", draws="host", checkerboard=True),
        # the batched workload: walkers of several lattice sizes in flight at once
        {"name": "many_6_10_14", "do": "many", "sizes": "6,10,14", "beta": 4.0, "dtau": 0.1, "nwrap": 5, "U": 6.0,
         "chains": 4, "form": "mixed"},
        # bins with equal-time scalar and lattice observables at every slice
        _sweep("square8_measure", "square", 8, 4.0, 0.1, 10, 4.0, 4, "mixed", measure=True),
        # one walker on the production lattice, plain and mixed form
        _sweep("square16_fp64", "square", 16, 4.0, 0.1, 10, 4.0, 1, "fp64"),
        _sweep("square16_mixed", "square", 16, 6.0, 0.1, 10, 4.0, 1, "mixed"),
        # plain form, several walkers, N_dim = 196 (no multiple of any tile)
        _sweep("square14_fp64_8", "square", 14, 4.0, 0.1, 10, 4.0, 8, "fp64"),
        # the benchmark's workload: 16 walkers, 16 x 16, beta = 10, mixed form (the largest)
        _sweep("square16_mixed_16", "square", 16, 10.0, 0.1, 10, 4.0, 16, "mixed"),
        # time-displaced Green functions every sweep, with their lattice bins: honeycomb (N_dim = 288)
        _sweep("honeycomb12_tau", "honeycomb", 12, 2.0, 0.05, 5, 5.0, 1, "mixed", ltau=1, measure=True),
        # Kondo lattice with the f-orbitals' interaction (vector vertices), plain form
        _sweep("kondo6_uf_tau", "kondo", 6, 3.0, 0.1, 10, 2.0, 4, "fp64", ltau=1, measure=True),
        # Kondo lattice, 144 + 144 orbitals, spin couplings alone, several walkers, mixed form
        _sweep("kondo12_tau", "kondo", 12, 2.0, 0.1, 10, 0.0, 4, "mixed", ltau=1, measure=True),
        # the stabilisation's Green function from UDV factors in host memory
        {"name": "cgr_256", "do": "cgr", "N": 256, "nvar": 2, "spread": 10.0},
    ]


def _cost(case):
    """Rough relative time of one pass, in products of N x N matrices of the mixed form."""
    if case["do"] == "many":
        return sum(_cost(dict(case, do="sweep", lattice="square", L1=int(s), L2=int(s), ltau=0))
                   for s in case["sizes"].split(","))
    if case["do"] != "sweep":
        return 0.0
    N, F, Lt = _sizes(case)
    c = case["chains"] * F * Lt * (float(N) ** 3 + 2e6 / case["chains"])
    if case["ltau"]:  # the 2N systems of the time-displaced functions, in either form
        return c * (30.0 if case["form"] == "fp64" else 18.0)
    return c * (4.0 if case["form"] == "fp64" else 1.0)


def draw(rng_):
    """One more case of the ranges above: every lattice, form, option; sizes from the smallest to
    the largest, even and odd, a cost of at most the largest listed one."""
    r = rng_
    while True:
        kind = r.choices(["square", "tau", "kondo", "many", "cgr", "decompose"], [8, 2, 2, 1, 1, 1])[0]
        form = r.choice(["fp64", "mixed"])
        chains = int(round(math.exp(r.uniform(0.0, math.log(16.0)))))
        if kind == "square":
            L1, L2 = r.randint(4, 16), r.randint(4, 16)
            U = round(r.uniform(2.0, 8.0), 2)
            cb = L1 % 2 == 0 and L2 % 2 == 0 and r.random() < 0.25
            case = _sweep("", "square", L1, r.choice([2.0, 3.0, 4.0, 6.0, 8.0, 10.0]), 0.1, 10 if U <= 4.0 else 5, U,
                          chains, form, r.choice(["device", "host"]), cb, 0,
                          r.random() < 0.3)
            case["L2"] = L2
        elif kind == "tau":
            case = _sweep("", r.choice(["square", "honeycomb"]), r.randint(3, 12), r.choice([1.0, 1.5, 2.0]), 0.05, 5,
                          5.0, min(chains, 4), form, "device", False, 1, True)
            case["L2"] = r.randint(3, 12)
        elif kind == "kondo":
            case = _sweep("", "kondo", r.randint(3, 12), r.choice([1.0, 1.7, 2.0, 3.0]), 0.1, r.choice([5, 10]),
                          r.choice([0.0, 2.0]), min(chains, 8), form, "device", False, r.choice([0, 1]), True)
            case["L2"] = r.randint(3, 12)
        elif kind == "many":
            case = {"do": "many", "sizes": ",".join(str(s) for s in sorted(r.sample(range(4, 17), r.randint(2, 5)))),
                    "beta": r.choice([2.0, 4.0, 6.0]), "dtau": 0.1, "nwrap": 5, "U": round(r.uniform(2.0, 8.0), 2),
                    "chains": min(chains, 6), "form": form}
        else:
            case = {"do": kind, "N": int(round(math.exp(r.uniform(math.log(16), math.log(400))))),
                    "spread": round(r.uniform(2.0, 12.0), 1)}
            if kind == "cgr":
                case["nvar"] = r.choice([1, 2])
            else:
                case["side"] = r.choice(["R", "L"])
        case.pop("name", None)
        if _cost(case) <= 0.8 * _cost(listed()[7]):
            return case


# ------------------------------------------------------------------------------------------------
# prepare / run
# ------------------------------------------------------------------------------------------------
@lru_cache(maxsize=64)
def _model_of(lattice, L1, L2, beta, dtau, nwrap, U, checkerboard):
    if lattice == "kondo":
        return model.kondo(L1, L2, JK=1.5, Uf=U, beta=beta, dtau=dtau, nwrap=nwrap)
    return model.hubbard(lattice, L1, L2, U=U, beta=beta, dtau=dtau, nwrap=nwrap, checkerboard=checkerboard)


def _model(case):
    return _model_of(case["lattice"], case["L1"], case["L2"], case["beta"], case["dtau"], case["nwrap"], case["U"],
                     case["checkerboard"])


def _sizes(case):
    """(N_dim, flavours, time slices)."""
    norb = 1 if case["lattice"] == "square" else 2
    return (case["L1"] * case["L2"] * norb, 1 if case["lattice"] == "kondo" else 2,
            int(round(case["beta"] / case["dtau"])))


@lru_cache(maxsize=16)
def _lattice(lattice, L1, L2):
    return lattice_obs.Lattice({"kondo": "bilayer_square"}.get(lattice, lattice), L1, L2)


def _chains(case, seed, first_chain=0):
    m = _model(case)
    C = case["chains"]
    ch = Chains(m, n_chains=C, precision=case["form"], ltau=case.get("ltau", 0))
    for c in range(C):
        ch.set_fields(c, rng.initial_fields(seed, first_chain + c, m.n_op, m.ltrot))
        ch.set_rng(c, seed + 1000 * first_chain, rng.sweep_counter_base(m.n_op, m.ltrot, 0))
    ch.init_state()
    if case.get("measure"):
        if case["lattice"] == "square":  # the library's scalar observables: no two-site vertices
            O = model.hopping_matrix("square", case["L1"], case["L2"]).real
            ch.set_scalar_obs(np.stack([O] * m.n_fl), np.full(m.ndim, case["U"]))
        ch.set_lattice_obs(_lattice(case["lattice"], case["L1"], case["L2"]))
    return ch


def _host_draws(case, seed):
    m = _model(case)
    return np.stack([rng.sweep_uniforms(seed, c, m.n_op, m.ltrot, 0) for c in range(case["chains"])])


def _udv_factors(N, spread, seed, count):
    """Factors as a run holds them: unitary U, descending scales over 10^(+-spread) and a well
    conditioned V (unit upper triangle with permuted columns), `count` of each."""
    r = np.random.default_rng(seed)
    out = []
    for _ in range(count):
        U = np.linalg.qr(r.standard_normal((N, N)) + 1j * r.standard_normal((N, N)))[0]
        D = 10.0 ** np.sort(r.uniform(-spread, spread, N))[::-1]
        V = np.eye(N) + np.triu(r.standard_normal((N, N)) + 1j * r.standard_normal((N, N)), 1) * (0.3 / math.sqrt(N))
        out += [U, D, V[:, r.permutation(N)]]
    return out


def prepare(case, seed):
    if case["do"] == "cgr":
        return {"case": case, "factors": _udv_factors(case["N"], case["spread"], seed, 2)}
    if case["do"] == "decompose":
        # U of decompose is the propagated product: no longer unitary
        r = np.random.default_rng([seed, 1])
        U, D, V = _udv_factors(case["N"], case["spread"], seed, 1)
        N = case["N"]
        U = (U + 0.3 * (r.standard_normal((N, N)) + 1j * r.standard_normal((N, N))) / math.sqrt(N))
        return {"case": case, "factors": [U, D, V]}
    if case["do"] == "many":
        hs = []
        for k, s in enumerate(case["sizes"].split(",")):
            sub = dict(case, do="sweep", lattice="square", L1=int(s), L2=int(s), checkerboard=False)
            hs.append(_chains(sub, seed, 100 * k))
        return {"case": case, "handles": hs}
    u = _host_draws(case, seed) if case["draws"] == "host" else None
    return {"case": case, "chains": _chains(case, seed), "draws": u}


def _by_chain(get, count):
    """Chain 0's array, and the other chains' in one."""
    rest = [get(c) for c in range(1, count)]
    return [get(0)] + ([np.stack(rest)] if rest else [])


def _readback(ch):
    return {"green": _by_chain(ch.green, ch.C), "fields": _by_chain(ch.fields, ch.C), "phase": ch.phase()}


def _lattice_bin(ch, kind, c):
    b = ch.lattice_obs(c, kind)["obs"]
    return np.concatenate([b[k].reshape(-1) for k in sorted(b)])


def _scalar_bin(ch, c):
    s = ch.scalar_obs(c)
    return np.array([s["kin"], s["pot"], s["part"], s["ener"]])


def run(state):
    case = state["case"]
    if case["do"] == "cgr":
        G, phase = cgr(case["nvar"], *state["factors"])
        return {"green": G, "phase": np.array([phase])}
    if case["do"] == "decompose":
        U, D, V = decompose(case["side"], *state["factors"])
        return {"U": U, "D": np.real(D), "V": V}
    if case["do"] == "many":
        sweep_many(state["handles"])
        return [_readback(h) for h in state["handles"]]
    ch = state["chains"]
    if case["measure"]:  # a bin of one sweep
        ch.reset_lattice_obs()
        if case["lattice"] == "square":
            ch.reset_scalar_obs()
    ch.sweep(state["draws"])
    out = _readback(ch)
    if case["measure"]:
        out["lattice"] = [_by_chain(lambda c, k=kind: _lattice_bin(ch, k, c), ch.C) for kind in range(1 + case["ltau"])]
        if case["lattice"] == "square":
            out["scalar"] = _by_chain(lambda c: _scalar_bin(ch, c), ch.C)
    return out


# ------------------------------------------------------------------------------------------------
# work: the bytes and operations of one pass
# ------------------------------------------------------------------------------------------------
def _sweep_work(case):
    """Operations (a complex multiply-add is 8): per slice and pass the two hopping products (one
    in checkerboard form: 16 per entry and bond side) and an accepted share of one half of the visits as
    rank-1 updates; propagation of U once per pass; per stabilisation two pivoted QRs with Q and the
    products and solves of G (about 59 N^3); time-displaced: four products per slice, and a 2N system per
    stabilisation.  Bytes: G and the fields in and out, the hopping matrices, draws and bins."""
    N, F, Lt = _sizes(case)
    C = case["chains"]
    nstm = -(-Lt // case["nwrap"])
    M = N if case["lattice"] != "kondo" else N // 2 + (N // 2 if case["U"] else 0)
    hop = 16.0 * N * N * 4 if case["checkerboard"] else 8.0 * N ** 3
    f = 2 * Lt * hop + Lt * hop + 2 * nstm * (14.7 + 44.0) * N ** 3 + 8.0 * N * N * M * Lt
    if case["ltau"]:
        f += 16.0 * Lt * N ** 3 + nstm * 8 * 40.0 * N ** 3
    b = C * (2 * F * N * N * 16 + 2 * M * Lt) + F * N * N * 16
    if case.get("draws") == "host":
        b += C * 6 * M * Lt * 8
    if case["measure"]:
        b += C * (5 if F == 2 else 3) * N * 2 * 16 * (1 + (Lt + 1) * case["ltau"])
    return {"bytes": float(b), "flops": C * F * f}


def work(case):
    if case["do"] == "cgr":
        N = case["N"]
        return {"bytes": 5.0 * N * N * 16, "flops": 44.0 * N ** 3}
    if case["do"] == "decompose":
        N = case["N"]
        return {"bytes": 4.0 * N * N * 16, "flops": 14.7 * N ** 3}
    if case["do"] == "many":
        ws = [_sweep_work(dict(case, lattice="square", L1=int(s), L2=int(s), checkerboard=False, ltau=0, measure=False))
              for s in case["sizes"].split(",")]
        return {k: sum(w[k] for w in ws) for k in ("bytes", "flops")}
    return _sweep_work(case)


# ------------------------------------------------------------------------------------------------
# exact: plain NumPy in 64 bits
# ------------------------------------------------------------------------------------------------
_ETA = {s: math.copysign(math.sqrt(2.0 * (3.0 + math.copysign(math.sqrt(6.0), abs(s) - 1.5))), s) for s in (-2, -1, 1, 2)}
_GAMMA = {s: 1.0 - math.copysign(math.sqrt(6.0), abs(s) - 1.5) / 3.0 for s in (-2, -1, 1, 2)}
_FLIP = {-2: (-1, 1, 2), -1: (1, 2, -2), 1: (2, -2, -1), 2: (-2, -1, 1)}


def _exact_hopping(case):
    """exp(-dtau T), exp(dtau T) and T of the lattice (t = 1, periodic), the dense exponential or, with
    checkerboard, the product of the bond exponentials family by family."""
    L1, L2 = case["L1"], case["L2"]
    cell = lambda a, b: (a % L1) + L1 * (b % L2)  # noqa: E731
    norb = 1 if case["lattice"] == "square" else 2
    T = np.zeros((L1 * L2 * norb,) * 2)
    fams = [[] for _ in range(4)]
    for n2 in range(L2):
        for n1 in range(L1):
            I = cell(n1, n2)
            if norb == 1:
                ends = [(I, cell(n1, n2 + 1)), (I, cell(n1 + 1, n2))]
                for b, e in enumerate(ends):
                    fams[(0 if (n1 + n2) % 2 == 0 else 2) + b].append(e)
            else:
                ends = [(2 * I, 2 * I + 1), (2 * I + 1, 2 * cell(n1, n2 + 1)), (2 * I, 2 * cell(n1 + 1, n2 - 1) + 1)]
            for i, j in ends:
                T[i, j] = T[j, i] = -1.0
    dt = case["dtau"]
    if case["checkerboard"]:
        B, Bi = np.eye(len(T)), np.eye(len(T))
        c, s = math.cosh(dt), math.sinh(dt)
        for fam in fams:
            E, Ei = np.eye(len(T)), np.eye(len(T))
            for i, j in fam:
                E[i, i] = E[j, j] = Ei[i, i] = Ei[j, j] = c
                E[i, j] = E[j, i] = s
                Ei[i, j] = Ei[j, i] = -s
            B, Bi = B @ E, Ei @ Bi
        return B, Bi, T
    w, Z = np.linalg.eigh(T)
    return (Z * np.exp(-dt * w)) @ Z.T, (Z * np.exp(dt * w)) @ Z.T, T


def _exact_green(blocks):
    """(1 + A_K ... A_1)^-1: the product factored block by block as Q D T with descending D."""
    N = len(blocks[0])
    Q, D, T = np.eye(N), np.ones(N), np.eye(N)
    for A in blocks:
        X = (A @ Q) * D
        p = np.argsort(-np.linalg.norm(X, axis=0), kind="stable")
        Q, R = np.linalg.qr(X[:, p])
        D = np.abs(np.diag(R))
        T = (R / D[:, None]) @ T[p]
    big, small = np.maximum(D, 1.0), np.minimum(D, 1.0)
    return np.linalg.solve(Q.T / big[:, None] + small[:, None] * T, Q.T / big[:, None])


def _exact_sweep(case, seed, chain, rng_seed):
    """One chain's sweep of the Mz Hubbard model: (G, fields, scalar sums)."""
    B, Bi, T = _exact_hopping(case)
    N, Lt, nw, dt, U = len(B), int(round(case["beta"] / case["dtau"])), case["nwrap"], case["dtau"], case["U"]
    g = math.sqrt(dt * U / 2.0)
    key = rng.uniforms
    f = np.where(key(seed, chain, 0, N * Lt).reshape(Lt, N) > 0.5, -1, 1)
    u = key(rng_seed, chain, N * Lt, 6 * N * Lt)
    ev = [lambda s, q=q: np.exp(q * g * np.vectorize(_ETA.get)(s)) for q in (1.0, -1.0)]  # E(s) per flavour
    stab = sorted(set(range(0, Lt, nw)) | {Lt})

    def product(flv, a, b):  # B_b ... B_{a+1}
        P = np.eye(N)
        for t in range(a, b):
            P = ev[flv](f[t])[:, None] * (B @ P)
        return P

    def fresh(t):  # G after slice t: (1 + B(t, 0) B(beta, t))^-1
        out = []
        for flv in (0, 1):
            cuts = [s for s in stab if s >= t]
            late = [product(flv, a, b) for a, b in zip(cuts, cuts[1:])]
            cuts = [s for s in stab if s <= t]
            early = [product(flv, a, b) for a, b in zip(cuts, cuts[1:])]
            # time runs 0 -> beta from the right: B(t, 0) stands left of B(beta, t)
            out.append(_exact_green(late + early))
        return out

    sums, I = np.zeros(4), np.eye(N)

    def measure(G):
        C = [I - x.T for x in G]
        kin = sum(float(np.sum(T * c)) for c in C)
        pot = float(np.sum(U * np.diag(C[0]) * np.diag(C[1])))
        part = sum(float(np.trace(c)) for c in C)
        sums[:] += (kin, pot, part, kin + pot)

    def visits(G, t, order, base):
        for k, n in enumerate(order):
            v = base + k
            so = int(f[t, n])
            sn = _FLIP[so][min(3, max(1, int(math.floor(u[3 * v] * 3.0 + 0.5 + 0.5)))) - 1]
            de = _ETA[sn] - _ETA[so]
            dl = [math.exp(g * de) - 1.0, math.exp(-g * de) - 1.0]
            ra = [1.0 + dl[k2] * (1.0 - G[k2][n, n]) for k2 in (0, 1)]
            if abs(ra[0] * ra[1] * _GAMMA[sn] / _GAMMA[so]) > u[3 * v + 2]:
                for k2 in (0, 1):
                    row = -G[k2][n].copy()
                    row[n] += 1.0
                    G[k2] -= np.outer(G[k2][:, n] * (dl[k2] / ra[k2]), row)
                f[t, n] = sn

    G = fresh(0)
    for t in range(Lt):
        for k in (0, 1):
            e = ev[k](f[t])
            G[k] = e[:, None] * (B @ G[k] @ Bi) / e[None, :]
        visits(G, t, range(N), t * N)
        if t + 1 in stab:
            G = fresh(t + 1)
        measure(G)
    for t in range(Lt, 0, -1):
        visits(G, t - 1, range(N - 1, -1, -1), Lt * N + (Lt - t) * N)
        for k in (0, 1):
            e = ev[k](f[t - 1])
            G[k] = Bi @ ((G[k] * e[None, :]) / e[:, None]) @ B
        if t > 1:
            measure(G)
            if t - 1 in stab:
                G = fresh(t - 1)
    return np.stack(fresh(0)).astype(complex), f.astype(np.int8), sums.astype(complex)


def _exact_qr(A):
    """LAPACK's pivoted QR (column norms downdated and recomputed exactly here): Q, R, pivots."""
    A = A.copy()
    N = len(A)
    piv = np.arange(N)
    Q = np.eye(N, dtype=complex)
    vs = []
    for j in range(N):
        p = j + int(np.argmax(np.sum(np.abs(A[j:, j:]) ** 2, axis=0)))
        A[:, [j, p]] = A[:, [p, j]]
        piv[[j, p]] = piv[[p, j]]
        a, x2 = A[j, j], float(np.sum(np.abs(A[j + 1:, j]) ** 2))
        if x2 == 0.0 and a.imag == 0.0:
            vs.append((None, 0.0))
            continue
        beta = -math.copysign(math.sqrt(abs(a) ** 2 + x2), a.real)
        tau = complex((beta - a.real) / beta, -a.imag / beta)
        v = np.concatenate([[1.0], A[j + 1:, j] / (a - beta)])
        A[j:, j:] -= np.conj(tau) * np.outer(v, v.conj() @ A[j:, j:])
        vs.append((v, tau))
    for j in range(N - 1, -1, -1):
        v, tau = vs[j]
        if v is not None:
            Q[j:] -= tau * np.outer(v, v.conj() @ Q[j:])
    return Q, np.triu(A), piv


def _exact_decompose(case, U, D, V):
    left = case["side"] == "L"
    Q, R, piv = _exact_qr(U * D)
    d = np.abs(np.diag(R))
    R = R / d[:, None]
    ph = np.prod(np.diag(R)) * round(np.linalg.det(np.eye(len(piv))[piv]))
    if left:
        ph = np.conj(ph)
    R[0] /= ph
    Q[:, 0] *= ph
    return {"U": Q, "D": d, "V": (V[:, piv] @ R.conj().T) if left else (R @ V[piv])}


def _exact_cgr(factors):
    UR, DR, VR, UL, DL, VL = factors
    br, bl = np.maximum(DR, 1.0), np.maximum(DL, 1.0)
    M = (UR.conj().T @ UL) / br[:, None] / bl + np.minimum(DR, 1.0)[:, None] * (VR @ VL) * np.minimum(DL, 1.0)
    return (UL / bl) @ np.linalg.solve(M, UR.conj().T / br[:, None])


def exact(case, seed):
    if case["do"] == "cgr":
        return {"green": _exact_cgr(_udv_factors(case["N"], case["spread"], seed, 2)), "phase": None}
    if case["do"] == "decompose":
        return _exact_decompose(case, *prepare(case, seed)["factors"])
    if case["do"] == "many":
        subs = [(k, dict(case, lattice="square", L1=int(s), L2=int(s), checkerboard=False))
                for k, s in enumerate(case["sizes"].split(","))]
        out = []
        for k, sub in subs:
            fit = sub["L1"] <= 10
            G, f, _ = _exact_sweep(sub, seed, 100 * k, seed + 100000 * k) if fit and k == 0 else (None, None, None)
            out.append({"green": [G, None], "fields": [f, None], "phase": None})
        return out
    N, F, Lt = _sizes(case)
    if case["lattice"] == "kondo" or N * N * N * Lt > 256 ** 3 * 60:  # two-site vertices; over 20 seconds
        return None
    G, f, s = _exact_sweep(case, seed, 0, seed)
    out = {"green": [G, None], "fields": [f, None], "phase": None}
    if case["measure"]:
        out["lattice"] = None
        if case["lattice"] == "square":
            out["scalar"] = [s, None]
    return out
