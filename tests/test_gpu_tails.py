"""A step's last operations (TFSF current points, NF2FF samples, probe ring) left
to the next step's first launch, against the f32 oracle (fields and ring bit for
bit): boxes clear of one another, and each overlap that keeps an operation at
its own place; one engine on the plane pipeline, and batches with UPML, with Mur
and with Mur beside dispersive media."""
import numpy as np
import pytest

from conftest import idx
from oracle.oracle import OracleEngine
from test_gpu_ade_adopt import media
from test_gpu_mur import SIX, faces
from test_gpu_parity import assert_bitexact, compare_fields, nf2ff_inputs, pml_region, rand_coeffs, seed_fields

pytestmark = pytest.mark.gpu
CASES = ["clear", "samples meet currents", "samples meet absorber", "currents meet absorber", "ring meets currents", "ring meets absorber"]


def build(cls, case, absorber, seed):
    """An engine and its oracle: a TFSF box inside an NF2FF surface inside the absorber, moved together by `case`."""
    N = (18, 17, 21)
    c = rand_coeffs(N, seed, pec_frac=0)
    g, o = cls(), OracleEngine(N, c, mode="f32")
    assert g.initGPU()
    g.init(N, c)
    g.setPlaneDepth(3)
    r = np.random.default_rng(seed)
    box = 3 if case == "currents meet absorber" else 4 if case == "samples meet currents" else 7
    nf = nf2ff_inputs(N, nfreq=2, inset=2 if case == "samples meet absorber" else 4)
    pts = [dict(field_idx=int(idx(n, x, y, z, *N)), delay_int=int(r.integers(0, 4)), delay_frac=float(r.random()), amp=0.3)
           for n in range(3) for x in (box, N[0] - 1 - box) for y in range(box, N[1] - box) for z in range(box, N[2] - box)]
    probes = [idx(2, 5, 6, 7, *N), idx(0, 12, 5, 6, *N)]
    if case == "ring meets currents":
        probes.append(pts[0]["field_idx"])
    if case == "ring meets absorber":
        probes += [idx(1, 8, 8, 0, *N), idx(0, 8, 8, 1, *N)]
    for e in (g, o):
        if absorber == "upml":
            e.configurePML([pml_region((0, 0, 0), (N[0], N[1], 3), 4), pml_region((0, 0, N[2] - 3), (N[0], N[1], 3), 5),
                            pml_region((0, 0, 3), (3, N[1], N[2] - 6), 6), pml_region((N[0] - 3, 0, 3), (3, N[1], N[2] - 6), 7)])
        else:
            e.configureMur(faces(N, 3, SIX))
        if absorber == "mur, media":
            e.configureLorentzADE(media(N, 3, False))
        e.configureTFSF(dict(signal=np.cos(np.arange(60) * 0.3).astype(np.float32), period=0, voltagePoints=pts[::3], currentPoints=pts))
        e.configureExcitation(dict(signal=np.sin(np.arange(30) * 0.4 + 0.1).astype(np.float32), delay=[0, 1], amp=[0.5, -0.7], dir=[2, 0],
                                   pos=[idx(0, 9, 9, 9, *N), pts[0]["field_idx"] % (N[0] * N[1] * N[2])], period=0))
        e.configureNF2FFAccumulation(nf)
    seed_fields(g, o, N, 6)
    g.configureProbeGatherBuffered(np.asarray(probes, np.uint32), 60, 1)
    return g, o, np.asarray(probes)


def oracle_steps(o, probes, steps, rows):
    for _ in range(steps):
        o.iterate(1)
        f = o.getFields()
        rows.append(np.stack([f["volt"][probes], f["curr"][probes]], -1).ravel())


def check(g, o, rows, what):
    compare_fields(g, o, what)
    assert_bitexact(g.readProbeGatherBuffered()["data"], np.concatenate(rows), what + " ring")
    ag, ao = g.readNF2FFAccumulation(True), o.readNF2FFAccumulation(True)
    for k in ("accumE", "accumH"):
        a, b = np.asarray(ag[k], np.float64), np.asarray(ao[k], np.float64)
        assert np.abs(a - b).max() <= 1e-6 * np.abs(b).max(), (what, k)


@pytest.mark.parametrize("case", CASES)
def test_one_engine(cuda_engine_cls, case):
    g, o, probes = build(cuda_engine_cls, case, "upml", 1)
    rows = []
    for steps in (1, 5, 37):
        g.iterate(steps)
        oracle_steps(o, probes, steps, rows)
        check(g, o, rows, "%s +%d" % (case, steps))


@pytest.mark.parametrize("absorbers", [("upml", "mur"), ("mur", "mur"), ("mur", "mur, media")])
@pytest.mark.parametrize("case", CASES)
def test_batch(cuda_engine_cls, case, absorbers):
    from efs_b200.engine import CudaBatch
    m = [build(cuda_engine_cls, case if i else "clear", a, i + 1) for i, a in enumerate(absorbers)]
    rows = [[], []]
    batch = CudaBatch([g for g, _, _ in m])
    for steps in (1, 5, 37):
        batch.iterate(steps)
        batch.sync()
        for i, (g, o, probes) in enumerate(m):
            oracle_steps(o, probes, steps, rows[i])
            check(g, o, rows[i], "%s %s +%d" % (case, absorbers[i], steps))
