"""The digit-sliced tensor-core products: what an output depends on, and how far it is off."""
import numpy as np
import pytest

from alf_gb300 import model as mdl, rng
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
