"""Small grids whose batches of steps run in one launch, bit for bit against the
f32 oracle: one cell, thin and padded rows, the largest grids of either
launch shape and the first beyond them, excitation entries that share a target, with and
without a period, more targets or probes than a CTA has threads, and batches
that end on either parity or span captured graphs."""
import numpy as np
import pytest

from oracle.oracle import OracleEngine
from test_gpu_parity import assert_bitexact, compare_fields, rand_coeffs, seed_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extra", ["none", "port", "period", "many targets", "many probes"])
@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("N", [(1, 1, 1), (2, 2, 2), (26, 11, 32), (5, 7, 9), (1, 40, 33), (300, 1, 5), (16, 32, 32), (16, 32, 33), (16, 64, 32), (16, 64, 33)])
def test_resident(cuda_engine_cls, N, dense, extra):
    if dense:
        c = rand_coeffs(N, 1)
    else:
        t = rand_coeffs((5, 1, 1), 1)
        c = dict(mat=np.random.default_rng(2).integers(0, 5, N).astype(np.uint32).ravel(),
                 table=np.concatenate([t[k].reshape(3, 5) for k in ("vv", "vi", "ii", "iv")]).T.astype(np.float32))
    g = cuda_engine_cls()
    assert g.initGPU()
    g.init(N, c)
    o = OracleEngine(N, c, mode="f32")
    n = N[0] * N[1] * N[2]
    r = np.random.default_rng(4)
    probes = None
    if extra != "none":
        k = 1600 if extra == "many targets" else 9
        pos = r.integers(0, n, k).astype(np.uint32)
        pos[-3:] = pos[:3]                                # entries that share a target (with the same component)
        comp = np.arange(k) % 3
        exc = dict(signal=np.sin(np.arange(30) * 0.4 + 0.1).astype(np.float32), delay=r.integers(0, 5, k), dir=comp, pos=pos,
                   amp=np.linspace(-0.7, 0.9, k).astype(np.float32), period=11 if extra == "period" else 0)
        g.configureExcitation(exc)
        o.configureExcitation(exc)
        probes = np.unique(np.concatenate([pos[:5] + n * comp[:5], r.integers(0, 3 * n, 1600 if extra == "many probes" else 6)])).astype(np.uint32)
    seed_fields(g, o, N, 6)
    if probes is not None:
        g.configureProbeGatherBuffered(probes, 60, 2)
    rows, done = [], 0
    for steps in (1, 2, 64, 69):
        g.iterate(steps)
        if probes is None:
            o.iterate(steps)
        for _ in range(steps if probes is not None else 0):
            o.iterate(1)
            done += 1
            if done % 2 == 0 and len(rows) < 60:
                f = o.getFields()
                rows.append(np.stack([f["volt"][probes], f["curr"][probes]], -1).ravel())
        compare_fields(g, o, "%s %s +%d" % (extra, N, steps))
    if probes is not None:
        assert_bitexact(g.readProbeGatherBuffered()["data"], np.concatenate(rows), "ring")
