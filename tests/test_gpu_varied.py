"""Core update of grids whose material changes at most planes (large tables),
bit for bit against the f32 oracle: scattered and graded materials beside
constant ones, odd sizes, UPML, Mur and a TFSF face, one engine and batches that
mix all kinds of members; and a step of scattered materials stays within what
reading their rows costs."""
import time

import numpy as np
import pytest

from conftest import idx
from oracle.oracle import OracleEngine
from test_gpu_mur import SIX, faces
from test_gpu_parity import compare_fields, pml_region, rand_coeffs, seed_fields

pytestmark = pytest.mark.gpu


def materials(N, kind, seed=1):
    r = np.random.default_rng(seed)
    x, y, z = np.meshgrid(*[np.arange(n, dtype=np.uint32) for n in N], indexing="ij")
    mat, rows = {"scattered": (r.integers(0, 1000, N), 1000), "graded": (x * N[2] + z, N[0] * N[2]),
                 "partly": (np.where(z < N[2] // 3, r.integers(0, 600, N), 0), 600),
                 "constant": (np.zeros(N, int), 448), "few": (r.integers(0, 5, N), 5)}[kind]
    t = rand_coeffs((rows, 1, 1), seed, pec_frac=0)
    return dict(mat=mat.astype(np.uint32).ravel(),
                table=np.concatenate([t[k].reshape(3, rows) for k in ("vv", "vi", "ii", "iv")]).T.astype(np.float32))


def build(cls, N, kind, what, depth, seed=1):
    c = rand_coeffs(N, seed, pec_frac=0) if kind == "dense" else materials(N, kind, seed)
    g, o = cls(), OracleEngine(N, c, mode="f32")
    assert g.initGPU()
    g.init(N, c)
    if depth:
        g.setPlaneDepth(depth)
    for e in (g, o):
        if what == "upml":
            e.configurePML([pml_region((0, 0, 0), (N[0], N[1], 3), 4), pml_region((0, 0, N[2] - 3), (N[0], N[1], 3), 5)])
        if what == "mur":
            e.configureMur(faces(N, 3, SIX))
        if what in ("face", "upml"):
            pts = [dict(field_idx=int(idx(n, p, q, N[2] // 2, *N)), delay_int=1, delay_frac=0.25, amp=0.7)
                   for n in (0, 1) for p in range(2, N[0] - 2) for q in range(2, N[1] - 2)]
            e.configureTFSF(dict(signal=np.cos(np.arange(20) * 0.3).astype(np.float32), period=0, voltagePoints=pts, currentPoints=[]))
    seed_fields(g, o, N, seed)
    return g, o


@pytest.mark.parametrize("depth", [3, 24])
@pytest.mark.parametrize("what", ["plain", "upml", "mur", "face"])
@pytest.mark.parametrize("kind", ["scattered", "graded", "partly", "constant", "few"])
@pytest.mark.parametrize("N", [(26, 17, 67), (5, 12, 130)])
def test_materials(cuda_engine_cls, N, kind, what, depth):
    g, o = build(cuda_engine_cls, N, kind, what, depth)
    for steps in (1, 4, 9):
        g.iterate(steps)
        o.iterate(steps)
        compare_fields(g, o, "%s %s %s +%d" % (N, kind, what, steps))


@pytest.mark.parametrize("what", ["plain", "upml", "mur", "face"])
def test_batch_of_all_kinds(cuda_engine_cls, what):
    from efs_b200.engine import CudaBatch
    m = [build(cuda_engine_cls, N, kind, what, 0, i + 1) for i, (N, kind) in enumerate(
        [((26, 17, 67), "scattered"), ((13, 12, 40), "few"), ((9, 14, 66), "dense"), ((20, 13, 64), "graded"), ((14, 15, 33), "constant")])]
    b = CudaBatch([g for g, _ in m])
    try:
        for steps, shape in ((1, None), (4, (5, 2)), (9, (24, 1))):
            if shape:
                b.setShape(*shape)
            b.iterate(steps)
            b.sync()
            for i, (g, o) in enumerate(m):
                o.iterate(steps)
                compare_fields(g, o, "%s member %d +%d" % (what, i, steps))
    finally:
        b.destroy()


@pytest.mark.parametrize("plane", [0, 5, 19])
def test_wait_runs_out_and_device_recovers(cuda_engine_cls, plane):
    """A plane whose loads are never issued (efs_debug_set_wait, as in test_gpu_timeout.py): the waits give up by design."""
    from efs_b200.engine import EfsError
    N = (20, 18, 24)
    g, o = build(cuda_engine_cls, N, "scattered", "plain", 0)
    g.debugSetWait(2_000_000, skip_plane=plane)
    g.iterate(1)
    with pytest.raises(EfsError) as err:
        g.sync()
    assert err.value.code == 5                # EFS_ERR_TIMEOUT
    g.debugSetWait()
    fresh, o = build(cuda_engine_cls, N, "scattered", "plain", 6)
    fresh.iterate(6)
    o.iterate(6)
    compare_fields(fresh, o, "after a timed-out wait on this device")


def test_scattered_materials_cost_their_rows(cuda_engine_cls):
    """150^3, core update alone: a row of every cell and side read from L2 each step moves 1.7 times a constant material's
    52 bytes a cell (the rows' two 32-byte sectors, halos included), so 2.8 times its time leaves room for their latency."""
    N, t = (150, 150, 150), {}
    r = np.random.default_rng(1)
    for rows in (1, 4096):
        g = cuda_engine_cls()
        assert g.initGPU()
        g.init(N, dict(mat=r.integers(0, rows, N).astype(np.uint32).ravel(), table=(0.3 + 0.1 * r.random((rows, 12))).astype(np.float32)))
        g.iterate(64)
        g.sync()
        best = 1e9
        for _ in range(6):
            t0 = time.perf_counter()
            g.iterate(256)
            g.sync()
            best = min(best, time.perf_counter() - t0)
        t[rows] = best
        g.destroy()
    assert t[4096] < 2.8 * t[1], t
