"""Far field at the edges of its blocks, chunks and slabs against the f64 oracle:
points one short of, on and past a record tile, axes with no points, points
grouped by normal axis or not, angle counts around a block, more angles than a
slab.  Bars as test_far_field_against_f64: 1e-4 of the largest field (f32 phase
and sums of at most 64 records before f64)."""
import numpy as np
import pytest

from oracle.oracle import far_field
from test_gpu_parity import nf2ff_inputs, rand_coeffs

pytestmark = pytest.mark.gpu


def run(cls, points, axes, ordered, nth, nph, freq=1.5e10, center=(6e-3, 5e-3, 7e-3)):
    N = (13, 11, 14)
    g = cls()
    assert g.initGPU()
    g.init(N, rand_coeffs(N, 1, pec_frac=0))
    r = np.random.default_rng(points + nph)
    cfg = nf2ff_inputs(N, nfreq=1)
    cells = np.stack([r.integers(1, n - 2, points) for n in N], axis=1).astype(np.uint32)
    cfg.update(surfaceIndices=cells.ravel(), numPoints=points)
    g.configureNF2FFAccumulation(cfg)
    n = 3 * N[0] * N[1] * N[2]
    g.uploadFields(r.standard_normal(n).astype(np.float32), r.standard_normal(n).astype(np.float32))
    g.iterate(17)
    acc = g.readNF2FFAccumulation(True)
    meta = np.zeros((points, 8), np.float32)
    meta[:, :3] = cells * 1e-3
    meta[:, 3] = r.choice(axes, points)
    if ordered:
        meta[:, 3].sort()
    meta[:, 4] = r.choice([-1.0, 1.0], points)
    meta[:, 5] = 1e-6
    th = np.linspace(0.1, 3.0, nth).astype(np.float32)
    ph = np.linspace(0.0, 6.2, nph).astype(np.float32)
    out = g.computeNF2FFfarField(dict(pointMeta=meta, theta=th, phi=ph, center=list(center), frequency=freq, radius=2.0,
                                      numPoints=points)).reshape(-1, 5)
    ref = far_field(acc["accumE"][0], acc["accumH"][0], meta, th, ph, freq, 2.0, center)
    assert np.abs(out[:, 1:] - ref[:, 1:]).max() <= 1e-4 * np.abs(ref[:, 1:]).max()
    assert np.abs(out[:, 0] - ref[:, 0]).max() <= 2e-4 * ref[:, 0].max()


@pytest.mark.parametrize("ordered", [True, False])
@pytest.mark.parametrize("points,axes", [(1, [2]), (255, [0, 1, 2]), (256, [1]), (257, [0, 2]), (1500, [0, 1, 2])])
@pytest.mark.parametrize("nth,nph", [(1, 1), (1, 127), (2, 64), (3, 43), (7, 61)])
def test_blocks_and_chunks(cuda_engine_cls, points, axes, ordered, nth, nph):
    run(cuda_engine_cls, points, axes, ordered, nth, nph)


def test_more_angles_than_a_slab(cuda_engine_cls):
    run(cuda_engine_cls, 9, [0, 1, 2], False, 601, 450)


def test_engine_repeats_and_changes_size(cuda_engine_cls):
    """The kept workspace serves calls of other sizes: each call as on a fresh engine."""
    N = (13, 11, 14)
    g = cuda_engine_cls()
    assert g.initGPU()
    g.init(N, rand_coeffs(N, 1, pec_frac=0))
    cfg = nf2ff_inputs(N, nfreq=2)
    g.configureNF2FFAccumulation(cfg)
    r = np.random.default_rng(3)
    n = 3 * N[0] * N[1] * N[2]
    g.uploadFields(r.standard_normal(n).astype(np.float32), r.standard_normal(n).astype(np.float32))
    g.iterate(9)
    meta = np.zeros((cfg["numPoints"], 8), np.float32)
    meta[:, :3] = cfg["surfaceIndices"].reshape(-1, 3) * 1e-3
    meta[:, 3] = r.integers(0, 3, cfg["numPoints"])
    meta[:, 4], meta[:, 5] = 1.0, 1e-6

    def call(nth, nph, fi):
        return g.computeNF2FFfarField(dict(pointMeta=meta, theta=np.linspace(0, 3, nth), phi=np.linspace(0, 6, nph),
                                           frequency=1e10, radius=1.0, numPoints=cfg["numPoints"], freqIndex=fi))
    first = call(5, 9, 0)
    call(40, 50, 1)
    assert np.array_equal(call(5, 9, 0), first)
