"""Digits of the far field against the f64 oracle.  A record's term is off by the
rounding of its phase (positions of at most 0.7 turns and three products in f32:
about 5e-7 rad), of the hardware sine and cosine (2^-21 each) and of the f32 sum
of at most 64 terms (about 4e-7): 1e-6 of the term, independent of the others, so
a field's error is 1e-6 of the fields' root mean square, and the largest of some
thousand values stays under ten times that."""
import numpy as np
import pytest

from oracle.oracle import far_field
from test_gpu_parity import nf2ff_inputs, rand_coeffs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("points,nth,nph", [(200, 7, 61), (3000, 19, 37)])
def test_digits(cuda_engine_cls, points, nth, nph):
    N = (13, 11, 14)
    g = cuda_engine_cls()
    assert g.initGPU()
    g.init(N, rand_coeffs(N, 1, pec_frac=0))
    r = np.random.default_rng(points)
    cells = np.stack([r.integers(1, n - 2, points) for n in N], axis=1).astype(np.uint32)
    cfg = nf2ff_inputs(N, nfreq=1)
    cfg.update(surfaceIndices=cells.ravel(), numPoints=points)
    g.configureNF2FFAccumulation(cfg)
    n = 3 * N[0] * N[1] * N[2]
    g.uploadFields(r.standard_normal(n).astype(np.float32), r.standard_normal(n).astype(np.float32))
    g.iterate(17)
    acc = g.readNF2FFAccumulation(True)
    meta = np.zeros((points, 8), np.float32)
    meta[:, :3], meta[:, 3] = cells * 1e-3, r.integers(0, 3, points)
    meta[:, 4], meta[:, 5] = r.choice([-1.0, 1.0], points), 1e-6
    th, ph = np.linspace(0.1, 3.0, nth).astype(np.float32), np.linspace(0.0, 6.2, nph).astype(np.float32)
    at, f = (6e-3, 5e-3, 7e-3), 1.5e10
    out = g.computeNF2FFfarField(dict(pointMeta=meta, theta=th, phi=ph, center=list(at), frequency=f, radius=2.0,
                                      numPoints=points)).reshape(-1, 5)
    ref = far_field(acc["accumE"][0], acc["accumH"][0], meta, th, ph, f, 2.0, at)
    assert np.abs(out[:, 1:] - ref[:, 1:]).max() <= 1e-5 * np.sqrt(np.mean(ref[:, 1:] ** 2))
