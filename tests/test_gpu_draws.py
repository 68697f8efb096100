"""The caller's own draws: what no generator gives, but an array can hold."""
import numpy as np
import pytest

from alf_gb300 import model as mdl, rng
from alf_gb300.sweep import FLAG_COMPLEX_ARITH, Chains

pytestmark = pytest.mark.gpu


# No weight is above a NaN, whichever its sign (0 / 0 on x86 has it set): every flip is rejected, in real and
# in complex arithmetic; a draw below zero accepts.
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("flags", [0, FLAG_COMPLEX_ARITH])
@pytest.mark.parametrize("value,accepted", [(np.nan, 0.0), (np.copysign(np.nan, -1.0), 0.0), (2.0 ** 300, 0.0),
                                            (np.inf, 0.0), (-1.0, 1.0), (-2.0 ** -1074, 1.0)])
def test_metropolis_draws_out_of_range(precision, flags, value, accepted):
    m = mdl.hubbard("square", 3, 3, U=1.0, beta=0.2, dtau=0.1, nwrap=1)
    g = Chains(m, precision=precision, flags=flags)
    g.set_fields(0, rng.initial_fields(31, 0, m.n_op, m.ltrot))
    g.init_state()
    u = rng.sweep_uniforms(31, 0, m.n_op, m.ltrot, 0).copy()
    u[2::3] = value
    g.set_recording(True)
    g.sweep(u[None])
    assert np.mean(g.record(0)["acc"]) == accepted
    g.close()


# weights that overflow (the factors exp(g dphi alpha) of the two flavours, each finite) or vanish: a complex
# product makes a NaN of the infinite ones, so none is accepted, in real arithmetic either
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("flags", [0, FLAG_COMPLEX_ARITH])
def test_infinite_weights_are_rejected(precision, flags):
    m = mdl.hubbard("square", 3, 3, U=1.0, beta=0.2, dtau=0.1, nwrap=1)
    pk = m.pack()
    g_ = pk["op_g"].real
    pk["op_type"][:] = 1  # fields +-1, phi(s) = s: every flip changes phi by 2
    pk["op_Eexp"][:, 0, :] = np.exp(g_[:, None] * np.arange(-2, 3))
    pk["op_alpha"][:] = 200.0 / g_  # exp(g dphi alpha) = exp(+-400)
    g = Chains(m, precision=precision, flags=flags)
    g._upload_vertices(-1, pk)
    f0 = rng.initial_fields(37, 0, m.n_op, m.ltrot)
    g.set_fields(0, f0)
    g.init_state()
    g.set_recording(True)
    g.sweep(rng.sweep_uniforms(37, 0, m.n_op, m.ltrot, 0)[None])
    assert not np.any(g.record(0)["acc"]) and np.array_equal(g.fields(0), f0)
    g.close()
