"""UPML z slabs of any thickness, listed row by row by the passes of the plane
pipeline, bit for bit against the f32 oracle: equal and unequal slabs, three over
the same rows, slabs that meet, alone and in a batch."""
import pytest

from oracle.oracle import OracleEngine
from test_gpu_parity import compare_fields, pml_region, rand_coeffs, seed_fields

pytestmark = pytest.mark.gpu
N = (6, 9, 70)


@pytest.mark.parametrize("batched", [False, True])
@pytest.mark.parametrize("slabs", [((0, 17), (53, 17)), ((0, 35), (35, 35)), ((0, 20), (49, 21)), ((2, 20), (22, 20), (50, 20)),
                                   ((0, 1), (69, 1))])
def test_thick_slabs(cuda_engine_cls, slabs, batched):
    from efs_b200.engine import CudaBatch
    g, o = cuda_engine_cls(), OracleEngine(N, rand_coeffs(N, 1), mode="f32")
    assert g.initGPU()
    g.init(N, rand_coeffs(N, 1))
    g.setPlaneDepth(3)
    for e in (g, o):
        e.configurePML([pml_region((0, 0, z), (N[0], N[1], n), i + 4) for i, (z, n) in enumerate(slabs)])
    seed_fields(g, o, N, 2)
    b = CudaBatch([g]) if batched else g
    for steps in (1, 4, 20):
        b.iterate(steps)
        b.sync()
        o.iterate(steps)
        compare_fields(g, o, "%s +%d" % (slabs, steps))
    if batched:
        b.destroy()
