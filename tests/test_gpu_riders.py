"""Excitation and probe samples that ride on the E sweep of small grids, bit for
bit against the f32 oracle: excitation targets at the ends of a block's run of
cells and more of them than a block has threads, probes on targets that Mur or
applied media write ahead of the sweep, sampling intervals, runs that end
anywhere, and operations that keep the excitation a launch of its own."""
import numpy as np
import pytest

from conftest import idx
from oracle.oracle import OracleEngine
from test_gpu_ade_adopt import media
from test_gpu_mur import SIX, faces
from test_gpu_parity import assert_bitexact, compare_fields, pml_region, rand_coeffs, seed_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("interval", [1, 3])
@pytest.mark.parametrize("targets", [1, 256, 257])
@pytest.mark.parametrize("case", ["plain", "mur", "ade", "upml", "tfsf"])
@pytest.mark.parametrize("N", [(4, 17, 66), (3, 9, 5)])
def test_riders(cuda_engine_cls, N, case, targets, interval):
    c = rand_coeffs(N, 1)
    g = cuda_engine_cls()
    assert g.initGPU()
    g.init(N, c)
    o = OracleEngine(N, c, mode="f32")
    n = N[0] * N[1] * N[2]
    r = np.random.default_rng(4)
    m = media(N, 3, False)
    pz = -(-N[2] // 4) * 4                                # a block takes 512 cells of a plane's padded rows
    ends = [x * N[1] * N[2] + y * N[2] + z for x in (0, N[0] - 1) for p in (0, 511, 512, 1023)
            for y, z in [divmod(p, pz)] if y < N[1] and z < N[2]]
    pos = np.concatenate([np.array(ends + [n - 1]), r.permutation(n)])[:targets].astype(np.uint32)
    if targets == 1:
        pos[:] = ends[1]
    comp = np.arange(len(pos)) % 3
    mur = faces(N, 5, SIX[:3])
    probes = np.unique(np.concatenate([pos[:20] + n * comp[:20], r.integers(0, 3 * n, 20),
                                       mur["normal_idx"][:3] if case == "mur" else [],
                                       m["orders"][0]["directions"][1]["pos_idx"][:3] + n if case == "ade" else []])).astype(np.uint32)
    for e in (g, o):
        e.configureExcitation(dict(signal=np.sin(np.arange(30) * 0.4 + 0.1).astype(np.float32), delay=np.arange(len(pos)) % 3,
                                   amp=np.linspace(-0.7, 0.9, len(pos)).astype(np.float32), dir=comp, pos=pos, period=0))
        if case == "mur":
            e.configureMur(mur)
        if case == "ade":
            e.configureLorentzADE(m)
        if case == "upml":
            e.configurePML([pml_region((0, 0, 0), (N[0], N[1], 3), 4)])
        if case == "tfsf":
            e.configureTFSF(dict(signal=np.cos(np.arange(20) * 0.3).astype(np.float32), period=0, currentPoints=[],
                                 voltagePoints=[dict(field_idx=int(pos[0] + n * comp[0]), delay_int=1, delay_frac=0.5, amp=0.6)]))
    seed_fields(g, o, N, 6)
    g.configureProbeGatherBuffered(probes, 40, interval)
    rows, done = [], 0
    for steps in (1, 5, 14):
        g.iterate(steps)
        for _ in range(steps):
            o.iterate(1)
            done += 1
            if done % interval == 0:
                f = o.getFields()
                rows.append(np.stack([f["volt"][probes], f["curr"][probes]], -1).ravel())
        compare_fields(g, o, "%s %s +%d" % (case, N, steps))
    got = g.readProbeGatherBuffered()
    assert got["numSamples"] == len(rows)
    assert_bitexact(got["data"], np.concatenate(rows), "ring %s" % case)
