"""The bench's roofline of the executed operations (no GPU): a bound on the measured steps."""
import json

import pytest

import bench
from alf_gb300 import model as mdl



# 16 x 16 Hubbard model, 16 chains, with the step times of this build and the accepted flips of its sweeps
# (acceptance 0.6 of 51,200 visits): the FP64 form's and the mixed form's step lie above their bound, where the reference's
# complex operations at the same peaks lie up to twice above them
@pytest.mark.parametrize("precision,ms", [("mixed", 307.6), ("fp64", 326.0)])
def test_bound_of_the_16x16_workload(precision, ms):
    m = mdl.config("hubbard16x16")
    g = [(m, 30000.0, 0, 16)]
    r = bench.executed_roofline(g, ms, precision, bench.FP64_DMMA_TFLOPS, 1900.0)
    assert 0.2 < r["frac"] <= 1.0
    n3 = 256.0 ** 3
    # QR, Q and solves a quarter of the complex count: 10.7 + 14.67 N^3 per stabilisation, 20 per flavour and sweep
    assert abs(r["flops_by_unit"]["fp64"] - 16 * 2 * 20 * (10.7 + 44.0 / 3.0) / 4.0 * n3) < 1e-9 * r["flops_per_step"]
    assert bench.sweep_roofline(m, 30000.0, 0, 16, ms, precision, bench.FP64_DMMA_TFLOPS, 1900.0)["frac"] > 1.0
    with pytest.raises(ValueError):
        bench.executed_roofline(g, 50.0, precision, bench.FP64_DMMA_TFLOPS, 1900.0)


def test_complex_models_and_small_grids():
    k = mdl.kondo(4, 4, JK=1.5, Uf=2.0, beta=2.0, dtau=0.1, nwrap=10)  # complex vertices: every operation executed
    r = bench.executed_roofline([(k, 100.0, 1, 2)], 1e6, "fp64", 1.0, 2000.0)
    ref = bench.reference_operations([(k, 100.0, 1, 2)], 1e6)
    assert abs(r["flops_per_step"] - ref["flops_per_step"]) < 1e-9 * ref["flops_per_step"]
    assert r["flops_by_unit"]["tensor"] == 0.0  # its products are too small for the tensor cores
    h = mdl.hubbard("square", 6, 6, beta=4.0)
    a, b = [(h, 100.0, 0, 3)], [(k, 100.0, 0, 2)]
    one = [bench.executed_roofline(x, 1e6, "mixed", 1.0, 2000.0)["t_roof_ms"] for x in (a, b)]
    assert abs(bench.executed_roofline(a + b, 1e6, "mixed", 1.0, 2000.0)["t_roof_ms"] - sum(one)) < 1e-12


def test_reported_beside_each_other():
    json.dumps(bench.executed_roofline([(mdl.config("hubbard4x4"), 100.0, 0, 1)], 4.5, "fp64", 1.0, 1900.0))
    assert set(bench.reference_operations([(mdl.config("hubbard4x4"), 100.0, 0, 1)], 4.5)) == {
        "flops_per_step", "flops_by_phase", "achieved_tflops"}


# digits as the library picks them, and none where it has none
@pytest.mark.parametrize("n,target,want", [(16, 54, (8, 7, 34)), (128, 54, (8, 7, 34)), (256, 54, (7, 8, 43)),
                                           (512, 54, (7, 8, 43)), (513, 54, (0, 0, 0)), (256, 61, (7, 9, 53)),
                                           (448, 61, (7, 9, 53)), (449, 61, (0, 0, 0))])
def test_digit_pairs(n, target, want):
    assert bench.digit_pairs(n, target) == want


def test_large_systems_on_the_fp64_pipes():
    m = mdl.hubbard("square", 22, 22, beta=0.2)  # N = 484: no 62-bit digits
    r = bench.executed_roofline([(m, 100.0, 0, 8)], 1e6, "fp64", 1.0, 1900.0)
    assert r["flops_by_unit"]["tensor"] == 0.0
    assert bench.executed_roofline([(m, 100.0, 0, 8)], 1e6, "mixed", 1.0, 1900.0)["flops_by_unit"]["tensor"] > 0.0
