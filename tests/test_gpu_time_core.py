"""Timing the core update of an engine that was reconfigured since its last step
(sweeps without UPML, whose kernels launch early, then with UPML, whose kernels
do not; and back) leaves its steps as they are, bit for bit against the f32
oracle."""
import pytest

from oracle.oracle import OracleEngine
from test_gpu_parity import compare_fields, pml_region, rand_coeffs, seed_fields

pytestmark = pytest.mark.gpu


def test_timing_after_reconfiguring(cuda_engine_cls):
    N = (20, 40, 66)
    c = rand_coeffs(N, 1)
    g, o = cuda_engine_cls(), OracleEngine(N, c, mode="f32")
    assert g.initGPU()
    g.init(N, c)
    seed_fields(g, o, N, 2)
    for regions in (None, [pml_region((0, 0, 0), (N[0], N[1], 3), 4)], [pml_region((0, 0, N[2] - 4), (N[0], N[1], 4), 5)]):
        if regions is not None:
            for e in (g, o):
                e.configurePML(regions)
        t = g.timeCore(20)
        assert t is not None
        g.iterate(6)
        o.iterate(6)
        compare_fields(g, o, "after timing")
