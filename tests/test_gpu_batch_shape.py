"""The shape of a batch's core update: the plan's own depth is among what the
autotuner times, so tuning never leaves a batch slower than it was, and depth 0
gives the choice back to the plan; every shape steps to the same bits."""
import time

import numpy as np
import pytest

from test_gpu_parity import assert_bitexact, rand_coeffs

pytestmark = pytest.mark.gpu
N = (400, 8, 64)      # one work tile per x-chunk: shallow chunks fill the device, the candidates' 8 planes and more do not


def batch(cls, members=1):
    from efs_b200.engine import CudaBatch
    es = []
    for i in range(members):
        g = cls()
        assert g.initGPU()
        g.init(N, rand_coeffs(N, i, pec_frac=0))
        n = 3 * N[0] * N[1] * N[2]
        r = np.random.default_rng(i)
        g.uploadFields(r.standard_normal(n).astype(np.float32), r.standard_normal(n).astype(np.float32))
        es.append(g)
    return CudaBatch(es), es


def fastest(b, runs=6, steps=640):
    t = []
    for _ in range(runs):
        b.sync()
        t0 = time.perf_counter()
        b.iterate(steps)
        b.sync()
        t.append(time.perf_counter() - t0)
    return min(t)


def test_tuning_never_loses_to_the_plan(cuda_engine_cls):
    b, es = batch(cuda_engine_cls)
    try:
        b.iterate(640)
        own = fastest(b)
        b.setShape(8)
        b.iterate(640)
        eight = fastest(b)
        assert eight > 1.2 * own          # the grid is one whose best depth is none of the candidates
        for steps in (16, 5):
            tuned = b.autotune(steps=steps)
            assert tuned["xchunk"] in (8, 16, 32, 64) and tuned["ctas_per_sm"] in (1, 2)
            b.iterate(640)
            assert fastest(b) < 1.15 * own, steps
        b.setShape(8)
        b.setShape(0)
        b.iterate(640)
        assert fastest(b) < 1.15 * own
    finally:
        b.destroy()
        for e in es:
            e.destroy()


def test_depth_of_the_plan_steps_to_the_same_bits(cuda_engine_cls):
    b, es = batch(cuda_engine_cls, 2)
    ref, rs = batch(cuda_engine_cls, 2)
    try:
        for shape in ((0, 1), (3, 2), (0, 2)):
            b.setShape(*shape)
            b.iterate(7)
            b.sync()
            ref.iterate(7)
            ref.sync()
            for e, r in zip(es, rs):
                f, q = e.getFields(), r.getFields()
                for k in ("volt", "curr"):
                    assert_bitexact(f[k], q[k], "%s %s" % (shape, k))
    finally:
        for x in (b, ref):
            x.destroy()
        for e in es + rs:
            e.destroy()
