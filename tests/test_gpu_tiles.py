"""The core update at the edges of its tiles, bit for bit against the f32 oracle.

With an explicit plane depth a grid runs the plane pipeline; without one a
grid that stays in L2 (or has dense coefficients) runs the E and H sweeps, one
thread per pair of z-adjacent cells in blocks of 256 pairs of an x-plane.

A tile is 64 (z) x 8 (y) cells over a chunk of x-planes; a thread owns two
z-adjacent cells and keeps their coefficients while their material repeats
along x.  Grids end one cell before, on and after a tile or a pair; materials
change along x cell by cell or never; UPML regions cover part of a chunk and
start between the cells of a pair.
"""
import numpy as np
import pytest

from oracle.oracle import OracleEngine
from test_gpu_parity import compare_fields, pml_region, rand_coeffs, seed_fields

pytestmark = pytest.mark.gpu


def engines(cls, N, coefficients, depth):
    g = cls()
    assert g.initGPU()
    g.init(N, coefficients)
    if depth:
        g.setPlaneDepth(depth)
    return g, OracleEngine(N, coefficients, mode="f32")


def materials(N, seed, run):
    """Material index that changes every `run` planes along x, differently for the two cells of a pair."""
    r = np.random.default_rng(seed)
    t = rand_coeffs((7, 1, 1), seed)
    table = np.concatenate([t[k].reshape(3, 7) for k in ("vv", "vi", "ii", "iv")]).T.astype(np.float32)
    ids = r.integers(0, 7, (N[0] // run + 1, N[1], N[2]))
    return dict(mat=np.repeat(ids, run, axis=0)[:N[0]].astype(np.uint32).ravel(), table=table)


@pytest.mark.parametrize("coef", ["dense", "every plane", "third plane"])
@pytest.mark.parametrize("depth", [None, 1, 2, 5])
@pytest.mark.parametrize("N", [(1, 8, 64), (2, 7, 63), (6, 9, 65), (11, 16, 66), (5, 1, 129), (9, 17, 2), (13, 8, 128)])
def test_tile_edges(cuda_engine_cls, N, depth, coef):
    c = rand_coeffs(N, 3) if coef == "dense" else materials(N, 4, 1 if coef == "every plane" else 3)
    g, o = engines(cuda_engine_cls, N, c, depth)
    seed_fields(g, o, N, 5)
    for steps in (1, 4):
        g.iterate(steps)
        o.iterate(steps)
        compare_fields(g, o, "%s depth %s %s +%d" % (N, depth, coef, steps))


@pytest.mark.parametrize("N", [(3, 16, 32), (2, 8, 63), (4, 13, 40), (3, 129, 4), (120, 120, 120), (121, 122, 120)])
def test_sweep_blocks_and_largest_grid(cuda_engine_cls, N):
    """Planes of exactly one block, one pair more, many rows; the largest grid that runs as sweeps and one above it."""
    g, o = engines(cuda_engine_cls, N, materials(N, 9, 3), None)
    regs = [pml_region((0, 0, 0), (N[0], 4, N[2]), 11), pml_region((1, 4, 0), (1, N[1] - 4, 3), 12)]
    for e in (g, o):
        e.configurePML(regs)
    seed_fields(g, o, N, 10)
    g.iterate(3)
    o.iterate(3)
    compare_fields(g, o, "sweep %s" % (N,))
    for r in range(2):
        assert np.array_equal(g.debugRead("pml_volt_flux", r), o.read("pml_volt_flux", r))
        assert np.array_equal(g.debugRead("pml_curr_flux", r), o.read("pml_curr_flux", r))


@pytest.mark.parametrize("depth", [None, 1, 4])
@pytest.mark.parametrize("boxes", [[((2, 0, 0), (3, 19, 70))], [((0, 0, 0), (12, 19, 9)), ((3, 2, 61), (5, 9, 9))],
                                   [((0, 7, 63), (12, 2, 2)), ((11, 0, 0), (1, 19, 30))]])
def test_upml_inside_tiles(cuda_engine_cls, boxes, depth):
    N = (12, 19, 70)
    g, o = engines(cuda_engine_cls, N, materials(N, 6, 2), depth)
    regs = [pml_region(s, n, 20 + i) for i, (s, n) in enumerate(boxes)]
    for e in (g, o):
        e.configurePML(regs)
    seed_fields(g, o, N, 7)
    g.iterate(6)
    o.iterate(6)
    compare_fields(g, o, "upml %s depth %s" % (boxes, depth))


def test_batch_tiles_sorted_by_kind(cuda_engine_cls):
    """A batch with enough plain tiles runs them apart from those that meet UPML regions: each member as alone."""
    from efs_b200.engine import CudaBatch
    sizes = [(40, 96, 130), (30, 80, 100)]
    pairs = []
    for i, N in enumerate(sizes):
        both = []
        for _ in range(2):
            g = cuda_engine_cls()
            assert g.initGPU()
            g.init(N, materials(N, 8 + i, 2))
            if i == 0:
                g.configurePML([pml_region((0, 0, 0), (40, 96, 6), 30), pml_region((0, 90, 6), (40, 6, 124), 31)])
            r = np.random.default_rng(40 + i)
            n = 3 * N[0] * N[1] * N[2]
            g.uploadFields(r.standard_normal(n).astype(np.float32), r.standard_normal(n).astype(np.float32))
            both.append(g)
        pairs.append(both)
    b = CudaBatch([p[0] for p in pairs])
    b.setShape(1)
    b.iterate(5)
    b.sync()
    for batched, alone in pairs:
        alone.iterate(5)
        f, h = batched.getFields(), alone.getFields()
        assert np.array_equal(f["volt"].view(np.uint32), h["volt"].view(np.uint32))
        assert np.array_equal(f["curr"].view(np.uint32), h["curr"].view(np.uint32))
    b.destroy()
