"""Applied ADE media computed ahead of the core update, bit for bit against the
f32 oracle: media that reach index 0 and the last lines, Drude and Lorentz
entries, runs that end anywhere, and cells that TFSF, an excitation, Mur, a
lumped element or a UPML region also touches (which keep the separate passes)."""
import numpy as np
import pytest

from conftest import idx
from oracle.oracle import OracleEngine
from test_gpu_mur import SIX, faces
from test_gpu_parity import assert_bitexact, compare_fields, pml_region, rand_coeffs, seed_fields

pytestmark = pytest.mark.gpu


def media(N, seed, share):
    """Two orders (Drude, Lorentz) on random cells, every component; share: the second order on cells of the first."""
    r = np.random.default_rng(seed)
    n = N[0] * N[1] * N[2]
    cells = np.flatnonzero(r.random(n) < 0.5).astype(np.uint32)
    first, second = cells[::2], cells[1::2]
    if share:
        second = first[:len(first) // 2]
    orders = []
    for c, lor in ((first, False), (second, True)):
        dirs = []
        for d in range(3):
            e = dict(dir=d, pos_idx=c, v_int_ADE=np.repeat(r.random(4).astype(np.float32), len(c) // 4 + 1)[:len(c)],
                     v_ext_ADE=(0.1 * r.random(len(c))).astype(np.float32) if d == 1 else np.full(len(c), 0.07, np.float32))
            if lor:
                e["v_Lor_ADE"] = np.full(len(c), 0.03 + 0.01 * d, np.float32)
            dirs.append(e)
        orders.append(dict(numCells=len(c), hasLorentz=lor, directions=dirs))
    return dict(orders=orders, apply=True)


@pytest.mark.parametrize("depth", [None, 3])
@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("case", ["alone", "shared", "tfsf", "excitation", "mur", "lumped", "upml"])
@pytest.mark.parametrize("N", [(9, 11, 66), (4, 3, 37)])
def test_applied_media(cuda_engine_cls, N, case, dense, depth):
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
    m = media(N, 3, case == "shared")
    cell = [int(v) for v in m["orders"][0]["directions"][0]["pos_idx"][[3, 10]]]
    for e in (g, o):
        if case == "upml":
            e.configurePML([pml_region((0, 0, 0), (N[0], N[1], 3), 4)])
        if case == "tfsf":
            n = N[0] * N[1] * N[2]
            pts = [dict(field_idx=k * n + cell[k], delay_int=1, delay_frac=0.5, amp=0.6) for k in range(2)]
            e.configureTFSF(dict(signal=np.cos(np.arange(20) * 0.3).astype(np.float32), period=0, voltagePoints=pts, currentPoints=[]))
        if case == "excitation":
            e.configureExcitation(dict(signal=np.sin(np.arange(30) * 0.4 + 0.1).astype(np.float32), delay=[0, 1], amp=[0.5, -0.7],
                                       dir=[2, 0], pos=cell, period=0))
        if case == "mur":
            e.configureMur(faces(N, 5, SIX[:3]))
        if case == "lumped":
            e.configureRLC(dict(elements=[dict(field_idx=cell[0], direction=1, type_flag=1, i2v=0.2, ilv=0.1, vvd=0.9, vv2=0.05,
                                               vj1=0.02, vj2=0.01, ib0=0.3, b1=0.1, b2=0.05)]))
        e.configureLorentzADE(m)
    seed_fields(g, o, N, 6)
    for steps in (1, 5, 14):
        g.iterate(steps)
        o.iterate(steps)
        compare_fields(g, o, "ade %s %s +%d" % (case, N, steps))
    assert np.isfinite(g.getFields()["volt"]).all()
