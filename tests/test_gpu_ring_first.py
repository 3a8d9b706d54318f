"""A probe ring configured before lumped elements (or before a call with none)
keeps its samples, against the f32 oracle: probes on targets that Mur or applied
media write ahead of the E sweep, in a UPML region, and on TFSF current points,
where the ring must not ride on the next step's first launch."""
import numpy as np
import pytest

from conftest import idx
from oracle.oracle import OracleEngine
from test_gpu_ade_adopt import media
from test_gpu_mur import SIX, faces
from test_gpu_parity import assert_bitexact, compare_fields, pml_region, rand_coeffs, seed_fields

pytestmark = pytest.mark.gpu
N = (12, 17, 21)


def build(cls, case, empty):
    c = rand_coeffs(N, 1, pec_frac=0)
    g, o = cls(), OracleEngine(N, c, mode="f32")
    assert g.initGPU()
    g.init(N, c)
    if case in ("absorber", "currents"):                  # the plane pipeline, whose UPML pass carries the samples
        g.setPlaneDepth(3)
    mur, med = faces(N, 5, SIX[:3]), media(N, 3, False)
    pts = [dict(field_idx=int(idx(n, x, y, 10, *N)), delay_int=1, delay_frac=0.5, amp=0.3) for n in (0, 1) for x in (5, 7) for y in (6, 9)]
    probes = [idx(2, 6, 8, 9, *N)]
    if case == "mur":
        probes += list(mur["normal_idx"][:5])
    if case == "media":
        probes += list(med["orders"][0]["directions"][1]["pos_idx"][:5] + N[0] * N[1] * N[2])
    if case == "absorber":
        probes += [idx(1, 8, 8, 0, *N), idx(0, 8, 8, 1, *N)]
    if case == "currents":
        probes.append(pts[0]["field_idx"])
    probes = np.unique(np.asarray(probes, np.uint32))
    seed_fields(g, o, N, 6)
    g.configureProbeGatherBuffered(probes, 60, 1)
    for e in (g, o):
        if case == "mur":
            e.configureMur(mur)
        if case == "media":
            e.configureLorentzADE(med)
        if case in ("absorber", "currents"):
            e.configurePML([pml_region((0, 0, 0), (N[0], N[1], 3), 4)])
        if case == "currents":
            e.configureTFSF(dict(signal=np.cos(np.arange(60) * 0.3).astype(np.float32), period=0, voltagePoints=[], currentPoints=pts))
        if not empty:
            at = idx(0, 6, 8, 9, *N)
            while case == "media" and any(at in d["pos_idx"] + d["dir"] * N[0] * N[1] * N[2] for d in
                                          [q for m in med["orders"] for q in m["directions"]]):
                at += 1                                   # a cell of its own: the media keep the form ahead of the sweep
            e.configureRLC(dict(elements=[dict(field_idx=int(at), direction=0, type_flag=0, i2v=0.3, ilv=0.2)]))
    if empty:
        assert g._lib.efs_configure_rlc(g._h, 0, None) == 0
    return g, o, probes


def check(g, o, probes, step, what):
    rows = []
    for steps in (1, 5, 18):
        step(steps)
        for _ in range(steps):
            o.iterate(1)
            f = o.getFields()
            rows.append(np.stack([f["volt"][probes], f["curr"][probes]], -1).ravel())
        compare_fields(g, o, "%s +%d" % (what, steps))
    assert_bitexact(g.readProbeGatherBuffered()["data"], np.concatenate(rows), what + " ring")


@pytest.mark.parametrize("empty", [False, True])
@pytest.mark.parametrize("case", ["mur", "media", "absorber", "currents"])
def test_ring_before_lumped_elements(cuda_engine_cls, case, empty):
    g, o, probes = build(cuda_engine_cls, case, empty)
    check(g, o, probes, g.iterate, case)


@pytest.mark.parametrize("case", ["mur", "absorber", "currents"])
def test_ring_before_no_elements_in_a_batch(cuda_engine_cls, case):
    from efs_b200.engine import CudaBatch
    g, o, probes = build(cuda_engine_cls, case, True)
    b = CudaBatch([g])
    try:
        def step(n):
            b.iterate(n)
            b.sync()
        check(g, o, probes, step, "batch " + case)
    finally:
        b.destroy()
