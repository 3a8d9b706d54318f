"""Large read-backs through the pinned ring: whole fields against plane copies,
for sizes around the staging threshold and a chunk, and from two threads."""
import threading

import numpy as np
import pytest

from test_gpu_parity import rand_coeffs

pytestmark = pytest.mark.gpu


def engine(cls, N, seed):
    g = cls()
    assert g.initGPU()
    g.init(N, rand_coeffs(N, seed))
    r = np.random.default_rng(seed)
    n = 3 * N[0] * N[1] * N[2]
    v, c = r.standard_normal(n).astype(np.float32), r.standard_normal(n).astype(np.float32)
    g.uploadFields(v, c)
    return g, v, c


@pytest.mark.parametrize("N", [(85, 64, 64), (86, 64, 64), (128, 64, 64), (128, 64, 68), (90, 61, 71)])
def test_fields_read_whole(cuda_engine_cls, N):
    g, v, c = engine(cuda_engine_cls, N, 1)
    for _ in range(2):
        f = g.getFields()
        assert np.array_equal(f["volt"], v) and np.array_equal(f["curr"], c)
    g.iterate(2)
    f = g.getFields()
    pv, pc = g.getPlanes(0, N[0])
    assert np.array_equal(f["volt"], pv.ravel()) and np.array_equal(f["curr"], pc.ravel())


def test_reads_from_two_threads(cuda_engine_cls):
    engines = [engine(cuda_engine_cls, (96, 80, 80), 2 + i) for i in range(2)]
    bad = []

    def read(g, v, c):
        for _ in range(6):
            f = g.getFields()
            if not (np.array_equal(f["volt"], v) and np.array_equal(f["curr"], c)):
                bad.append(1)
    th = [threading.Thread(target=read, args=e) for e in engines]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not bad
