"""Mur entries computed ahead of the core update and entries left to the three
passes around it, bit for bit against the f32 oracle: entries that share
cells, targets and shifted cells that UPML, TFSF, an excitation or a periodic
axis touch, and grids so thin that opposite faces meet."""
import numpy as np
import pytest

from conftest import idx
from oracle.oracle import OracleEngine
from test_gpu_parity import assert_bitexact, compare_fields, pml_region, rand_coeffs, seed_fields

pytestmark = pytest.mark.gpu


def faces(N, seed, which):
    """Mur entries of the faces `which` ((axis, 'lo'|'hi'), ...), in the order given: {coeff, normal_idx, shifted_idx}."""
    r = np.random.default_rng(seed)
    nrm, shf = [], []
    for a, side in which:
        line, shift = (0, 1) if side == "lo" else (N[a] - 1, N[a] - 2)
        for n in ((a + 1) % 3, (a + 2) % 3):
            g = np.meshgrid(*[np.array([line]) if b == a else np.arange(N[b]) for b in range(3)], indexing="ij")
            p = [x.ravel() for x in g]
            q = [np.full_like(p[0], shift) if b == a else p[b] for b in range(3)]
            nrm.append(idx(n, *p, *N))
            shf.append(idx(n, *q, *N))
    nrm, shf = np.concatenate(nrm), np.concatenate(shf)
    return dict(coeff=(0.5 * r.random(len(nrm)) - 0.1).astype(np.float32), normal_idx=nrm, shifted_idx=shf)


SIX = [(a, s) for a in range(3) for s in ("lo", "hi")]
CASES = ["plain", "upml", "tfsf", "excitation", "periodic", "pile"]


@pytest.mark.parametrize("depth", [None, 3])
@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("N", [(9, 17, 66), (2, 3, 5), (12, 2, 33)])
def test_mur_split(cuda_engine_cls, N, case, dense, depth):
    if dense:
        c = rand_coeffs(N, 1)
    else:
        r = np.random.default_rng(2)
        t = rand_coeffs((5, 1, 1), 1)
        c = dict(mat=r.integers(0, 5, N).astype(np.uint32).ravel(),
                 table=np.concatenate([t[k].reshape(3, 5) for k in ("vv", "vi", "ii", "iv")]).T.astype(np.float32))
    g = cuda_engine_cls()
    assert g.initGPU()
    g.init(N, c)
    if depth:
        g.setPlaneDepth(depth)
    o = OracleEngine(N, c, mode="f32")
    m = faces(N, 3, SIX)
    x, y, z = N[0] - 1, N[1] // 2, N[2] // 2
    if case == "pile":               # one target written many times: more entries than a group takes
        m = {k: np.concatenate([v] + [v[7:8]] * 12) for k, v in m.items()}
        m["coeff"][-12:] = np.linspace(-0.3, 0.4, 12, dtype=np.float32)
    for e in (g, o):
        if case == "upml":
            e.configurePML([pml_region((0, 0, 0), (N[0], N[1], 2), 4)])
        if case == "tfsf":           # targets on a Mur target, on a shifted cell, elsewhere
            pts = [dict(field_idx=int(f), delay_int=1, delay_frac=0.25, amp=0.7) for f in
                   (idx(1, x, y, z, *N), idx(2, 1, y, z, *N), idx(0, 0, y, z, *N), idx(2, x, 0, z, *N))]
            e.configureTFSF(dict(signal=np.cos(np.arange(20) * 0.3).astype(np.float32), period=0, voltagePoints=pts,
                                 currentPoints=pts[:1]))
        if case == "excitation":     # on a Mur target (the apply step wins) and on a shifted cell (read before)
            pos = [idx(0, x, y, z, *N), idx(0, 1, y, z, *N), idx(0, 0, 0, z, *N)]
            e.configureExcitation(dict(signal=np.sin(np.arange(30) * 0.4 + 0.1).astype(np.float32), delay=[0, 1, 0],
                                       amp=[0.5, -0.7, 0.9], dir=[2, 2, 1], pos=pos, period=0))
        if case == "periodic":
            e.configurePBC(dict(axes=[dict(axis=1, phase=0.0)]))
        e.configureMur(m)
    seed_fields(g, o, N, 5)
    for steps in (1, 4, 20):
        g.iterate(steps)
        o.iterate(steps)
        compare_fields(g, o, "mur %s %s +%d" % (case, N, steps))
    assert_bitexact(g.debugRead("mur_saved"), o.read("mur_saved"), "mur_saved %s" % case)
    # reconfigured: the adopt bits follow the new entries
    m2 = faces(N, 6, SIX[:2])
    for e in (g, o):
        e.configureMur(m2)
    g.iterate(3)
    o.iterate(3)
    compare_fields(g, o, "mur again %s" % case)
