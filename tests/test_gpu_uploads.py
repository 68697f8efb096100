"""Uploads to a handle that has run: the arithmetic follows the vertices that it holds."""
import numpy as np
import pytest

from alf_gb300 import _lib, model as mdl, rng
from alf_gb300.sweep import Chains

pytestmark = pytest.mark.gpu


def _complex_tables(m):
    """The model's tables with imaginary couplings."""
    pk = m.pack()
    pk["op_g"] = pk["op_g"] * 1j
    pk["op_Eexp"] = np.exp(1j * np.log(pk["op_Eexp"].real))
    return pk


def _run(g, m):
    g.set_fields(0, rng.initial_fields(29, 0, m.n_op, m.ltrot))
    g.set_rng(0, 29, rng.sweep_counter_base(m.n_op, m.ltrot, 0))
    g.init_state()
    for _ in range(2):  # captured, replayed
        g.sweep(None)
    return g.green(0), g.fields(0), g.phase()


def _same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.fixture(params=["fp64", "mixed"])
def handles(request):
    m = mdl.hubbard("square", 6, 6, U=4.0, beta=0.8, dtau=0.1, nwrap=4)
    g, ref = Chains(m, precision=request.param), Chains(m, precision=request.param)
    yield m, g, _run(ref, m)
    g.close()
    ref.close()


# the real and the complex kernels round differently, so equal bits say which of them ran
def test_a_refused_upload_changes_nothing(handles):
    m, g, want = handles
    pk = _complex_tables(m)
    pk["op_g"][-1] = np.nan
    with pytest.raises(_lib.AlfGpuError) as e:
        g._upload_vertices(-1, pk)
    assert e.value.code == 6
    assert _same(_run(g, m), want)


def test_real_vertices_in_place_of_complex_ones(handles):
    m, g, want = handles
    g._upload_vertices(-1, _complex_tables(m))
    assert not np.array_equal(_run(g, m)[0], want[0])
    g._upload_vertices(-1, m.pack())
    assert _same(_run(g, m), want)
