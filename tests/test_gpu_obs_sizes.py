"""The device-side observables at sizes around their splits (cells around 32 and 128, two
orbitals per cell, one CTA and a cluster of eight per chain), in real and complex arithmetic,
three chains per handle, against the host restatements fed the same sweep's callbacks: the same
G in another summation order, 1e-10 relative to the largest entry."""
import numpy as np
import pytest

from alf_gb300 import lattice_obs as lo, model as mdl, rng
from alf_gb300.sweep import FLAG_COMPLEX_ARITH, Chains
from test_gpu_latt_obs import _close
from test_gpu_obs import _host_sums

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [0, FLAG_COMPLEX_ARITH])
@pytest.mark.parametrize("lattice,L1,L2", [("square", 2, 2), ("square", 8, 4), ("square", 11, 3), ("square", 12, 11),
                                           ("honeycomb", 3, 2), ("honeycomb", 8, 9), ("kondo", 3, 2)])
def test_observables_match_host_sums(lattice, L1, L2, flags):
    if lattice == "kondo":  # one flavour, complex vertices
        m, latt = mdl.kondo(L1, L2, JK=1.5, Uf=2.0, beta=0.2, dtau=0.1, nwrap=1), "bilayer_square"
    else:
        m, latt = mdl.hubbard(lattice, L1, L2, U=4.0, beta=0.2, dtau=0.1, nwrap=1), lattice
    latt = lo.Lattice(latt, L1, L2)
    g = Chains(m, n_chains=3, ltau=1, flags=flags)
    for c in range(3):
        g.set_fields(c, rng.initial_fields(21, c, m.n_op, m.ltrot))
    g.init_state()
    g.set_lattice_obs(latt)
    rs = np.random.default_rng(4)
    H = rs.standard_normal((m.n_fl, m.ndim, m.ndim))
    U = rs.standard_normal(m.ndim)
    if lattice != "kondo":  # scalar observables are the Hubbard-type models'
        g.set_scalar_obs(H, U)
    u = np.stack([rng.sweep_uniforms(21, c, m.n_op, m.ltrot, 0) for c in range(3)])
    eq, tau = g.sweep(u, measure=True)
    for c in range(3):
        eh = lo.EqualTimeObs(latt, n_sun=m.n_sun, n_fl=m.n_fl)
        th = lo.TimeDisplacedObs(latt, n_sun=m.n_sun, ntau=m.ltrot + 1, n_fl=m.n_fl)
        mine = [(cc, G, ph) for cc, nt, G, ph in eq if cc == c]
        for _, G, ph in mine:
            eh.measure(G, ph)
        for cc, nt, q, ph in tau:
            if cc == c:
                th.measure(nt, *q, ph)
        for kind, host in ((0, eh.bin()), (1, th.bin())):
            dev = g.lattice_bin(c, kind)
            for k in host:
                assert _close(dev[k]["latt"], host[k]["latt"]), (kind, k)
                assert _close(dev[k]["latt0"], host[k]["latt0"]), (kind, k)
                assert dev[k]["sign"] == host[k]["sign"]
        if lattice == "kondo":
            continue
        d, ref = g.scalar_obs(c), _host_sums(mine, H, U, m.n_sun)
        assert d["count"] == ref["count"] and d["sign"] == ref["sign"]
        for k in ("kin", "pot", "part", "ener"):
            assert abs(d[k] - ref[k]) <= 1e-10 * max(1.0, abs(ref[k])), k
    g.close()
