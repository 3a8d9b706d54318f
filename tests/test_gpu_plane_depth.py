"""Plane depth 0 gives the choice of form and depth back to the engine: a small
grid runs all steps of a batch in one launch again, a larger one as sweeps, bit
for bit against the f32 oracle through every change."""
import pytest

from oracle.oracle import OracleEngine
from test_gpu_parity import compare_fields, pml_region, rand_coeffs, seed_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,upml,launches", [((6, 9, 12), False, 1), ((20, 40, 66), False, 2), ((6, 9, 12), True, 2)])
def test_depth_given_back(cuda_engine_cls, N, upml, launches):
    g, o = cuda_engine_cls(), OracleEngine(N, rand_coeffs(N, 1), mode="f32")
    assert g.initGPU()
    g.init(N, rand_coeffs(N, 1))
    if upml:
        for e in (g, o):
            e.configurePML([pml_region((0, 0, 0), (N[0], N[1], 3), 4)])
    seed_fields(g, o, N, 2)
    seen = []
    for depth in (None, 32, 3, 0):
        if depth is not None:
            g.setPlaneDepth(depth)
        seen.append(g.kernelsPerStep())
        g.iterate(7)
        o.iterate(7)
        compare_fields(g, o, "%s depth %s" % (N, depth))
    assert seen[0] == seen[3] == launches and seen[1] == seen[2], seen
    with pytest.raises(Exception):
        g.setPlaneDepth(65536)
