"""Device memory of a handle: what the FP64 form takes for products on the tensor cores."""
import numpy as np
import pytest

from alf_gb300 import model as mdl, rng
from alf_gb300.sweep import FLAG_NO_TENSOR_GEMM, Chains

pytestmark = pytest.mark.gpu
MB = 1 << 20


def _free():
    torch = pytest.importorskip("torch")
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _handle(m, chains, flags):
    """A ready handle and the memory it took."""
    before = _free()
    g = Chains(m, n_chains=chains, flags=flags)
    for c in range(chains):
        g.set_fields(c, rng.initial_fields(23 + c, c, m.n_op, m.ltrot))
        g.set_rng(c, 23 + c, rng.sweep_counter_base(m.n_op, m.ltrot, 0))
    g.init_state()
    g.sweep(None)
    return g, before - _free()


# no product of these handles is worth the tensor cores, so the handle has no buffers for them (digit slices
# would be some hundred times G): as much memory as with FLAG_NO_TENSOR_GEMM, to an allocation's rounding
@pytest.mark.parametrize("L,chains", [(3, 400), (4, 200), (8, 4)])
def test_no_tensor_buffers_where_they_do_not_pay(L, chains):
    m = mdl.hubbard("square", L, L, U=4.0, beta=0.4, dtau=0.1, nwrap=2)
    _handle(m, chains, FLAG_NO_TENSOR_GEMM)[0].close()  # kernels loaded, once
    took = []
    for flags in (FLAG_NO_TENSOR_GEMM, 0):
        g, n = _handle(m, chains, flags)
        took.append(n)
        g.close()
    assert took[1] <= took[0] + 4 * MB, took


# products that pay, in memory that holds the handle but not their buffers: the FP64 pipes do them
def test_without_room_for_tensor_buffers():
    torch = pytest.importorskip("torch")
    m = mdl.hubbard("square", 8, 8, U=4.0, beta=0.4, dtau=0.1, nwrap=2)
    took, G = [], []
    for rep in range(2):
        took = []
        for flags in (FLAG_NO_TENSOR_GEMM, 0):
            g, n = _handle(m, 128, flags)
            took.append(n)
            G.append(g.green(5))
            g.close()
    assert took[1] >= took[0] + 64 * MB, took
    rest = torch.empty(_free() - (took[0] + took[1]) // 2, dtype=torch.uint8, device="cuda:0")
    try:
        assert took[0] + 16 * MB <= _free() <= took[1] - 16 * MB
        g, _ = _handle(m, 128, 0)
        got = g.green(5)
        g.close()
    finally:
        del rest
        torch.cuda.empty_cache()
    assert np.array_equal(got, G[0]) and not np.array_equal(G[0], G[1])
