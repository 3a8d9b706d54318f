"""Mur entries of the three passes (pre, post, apply) in batches, bit for bit
against the f32 oracle: members that have such entries and neither an excitation
nor TFSF points in the point pass, alone and beside members that have a port."""
import numpy as np
import pytest

from conftest import idx
from oracle.oracle import OracleEngine
from test_gpu_mur import SIX, faces
from test_gpu_parity import assert_bitexact, compare_fields, pml_region, rand_coeffs, seed_fields

pytestmark = pytest.mark.gpu
N = (9, 17, 21)


def member(cls, case, seed):
    g, o = cls(), OracleEngine(N, rand_coeffs(N, seed), mode="f32")
    assert g.initGPU()
    g.init(N, rand_coeffs(N, seed))
    m = faces(N, 3, SIX)
    if case == "pile":               # one target written by more entries than a group takes
        m = {k: np.concatenate([v] + [v[7:8]] * 12) for k, v in m.items()}
        m["coeff"][-12:] = np.linspace(-0.3, 0.4, 12, dtype=np.float32)
    for e in (g, o):
        if case == "absorber":       # Mur entries in UPML cells
            e.configurePML([pml_region((0, 0, 0), (N[0], N[1], 3), 4)])
        if case == "sheet":          # a TFSF sheet that meets the Mur faces, all of it applied in the core update
            pts = [dict(field_idx=int(idx(n, x, y, 10, *N)), delay_int=1, delay_frac=0.25, amp=0.7)
                   for n in (0, 1) for x in range(N[0]) for y in range(N[1])]
            e.configureTFSF(dict(signal=np.cos(np.arange(20) * 0.3).astype(np.float32), period=0, voltagePoints=pts, currentPoints=[]))
        if case == "port":           # no Mur entry near it takes the three passes
            e.configureExcitation(dict(signal=np.sin(np.arange(30) * 0.4 + 0.1).astype(np.float32), delay=[0], amp=[0.5], dir=[2],
                                       pos=[idx(0, 4, 8, 9, *N)], period=0))
        e.configureMur(m)
    seed_fields(g, o, N, seed)
    return g, o


@pytest.mark.parametrize("beside", [(), ("port",)])
@pytest.mark.parametrize("case", ["absorber", "sheet", "pile"])
def test_mur_post_in_batches(cuda_engine_cls, case, beside):
    from efs_b200.engine import CudaBatch
    m = [member(cuda_engine_cls, c, i + 1) for i, c in enumerate((case,) + beside)]
    b = CudaBatch([g for g, _ in m])
    try:
        for steps in (1, 4, 20):
            b.iterate(steps)
            b.sync()
            for g, o in m:
                o.iterate(steps)
                compare_fields(g, o, "%s %s +%d" % (case, beside, steps))
        for g, o in m:
            assert_bitexact(g.debugRead("mur_saved"), o.read("mur_saved"), "mur_saved %s" % case)
    finally:
        b.destroy()
        for g, _ in m:
            g.destroy()
