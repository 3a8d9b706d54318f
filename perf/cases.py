"""Performance cases: the work a user of the engine has it do, through its public calls.

A case is a plain dict.  `kind` says which calls it makes:

* "solve"    one engine (`CudaEngine`): `steps` timesteps, the energy, the
             probe ring, the NF2FF accumulators, the fields;
* "batch"    several engines advanced together (`CudaBatch`): `steps`
             timesteps of every member, then its probe rings and fields;
* "farfield" the far field of one frequency from the NF2FF accumulators.

Every solve starts from the fields of a solve under way (random values of a
field's scale, drawn on the GPU), with material boxes, dispersive spheres and
the pulse drawn from the seed, so no part of the grid is empty or constant.
"""
import functools
import math

import numpy as np
import torch

from efs_b200 import opgen, workloads
from efs_b200.engine import CudaBatch, CudaEngine

DELTA = 0.5e-3              # cell size of the uniform meshes (the headline workload's)
F0, FC = 10e9, 5e9          # pulse band
Z0 = 376.73031346177066
C0 = 299792458.0

# The defaults of a solve.
#   coef   "table": material index + table; "arrays": the dense vv/vi/ii/iv arrays of a graded mesh
#          (mild: uniform core, the engine's table form); "unique": the same with every spacing its own
#          (the engine keeps the dense arrays)
#   pml    UPML thickness in lines (0: none) on "faces" "z" or "all"
#   mur    Mur ABC faces: "none", "xy", "five" (all but zmin, a ground plane), "six"
#   source "port": additive z column + voltage and current probes; "tfsf": plane wave at `angle` degrees + NF2FF
#          with `nfreq` frequencies
#   ade    "none", "state" (the reference's form), "apply" (dispersion acts on the fields)
BASE = dict(kind="solve", coef="table", pml=0, faces="all", mur="none", source="port", angle=0.0, nfreq=0, ade="none",
            interval=3)


def _solve(name, grid, steps, **more):
    d = dict(BASE, name=name, nx=grid[0], ny=grid[1], nz=grid[2], steps=steps)
    d.update(more)
    return d


def listed():
    return [
        # the smallest call: a PEC cavity of the resonator fixture's size, one energy check's steps
        _solve("cavity_26x11x32", (26, 11, 32), 100),
        # an antenna in open space: the dipole fixture's grid, Mur on six faces
        _solve("dipole_81_mur", (81, 81, 81), 100, mur="six", interval=21),
        # the patch antenna's grid: graded mesh given as arrays, UPML on all faces, probes every step
        _solve("patch_86x87x71_upml", (86, 87, 71), 100, coef="arrays", pml=8, interval=1),
        # a graded mesh whose cells all differ (dense coefficients), odd sizes, ground plane and Mur
        _solve("graded_121x109x97_dense", (121, 109, 97), 100, coef="unique", mur="five", interval=5),
        # scattering solves: plane wave, UPML on z, Mur on x and y, three NF2FF frequencies
        _solve("scatter_256", (256, 256, 256), 200, pml=8, faces="z", mur="xy", source="tfsf", nfreq=3),
        # the headline size
        _solve("scatter_512", (512, 512, 512), 200, pml=8, faces="z", mur="xy", source="tfsf", nfreq=3),
        # dispersive spheres, UPML on all faces, oblique wave, five frequencies: the reference's state-only form
        _solve("dispersive_320_state", (320, 320, 160), 100, pml=8, source="tfsf", angle=30.0, nfreq=5, ade="state"),
        # and with the media acting on the fields
        _solve("dispersive_200_apply", (200, 200, 100), 100, pml=8, source="tfsf", angle=30.0, nfreq=5, ade="apply"),
        # a parameter sweep: stub-filter grids (lumped port, Mur on five faces) advanced together
        dict(name="sweep_32_ports", kind="batch", count=32, lo=60, hi=180, tfsf=0.0, steps=64),
        # the served mix at its small end: ports, and plane-wave jobs with NF2FF
        dict(name="served_16_mixed", kind="batch", count=16, lo=40, hi=96, tfsf=0.3, steps=64),
        # far field of an antenna on the runner's grid (3 and 5 degrees), after a small solve
        dict(name="farfield_runner", kind="farfield", nx=86, ny=87, nz=71, inset=10, nth=61, nph=73),
        # and on a 1 degree grid after a large one
        dict(name="farfield_fine_256", kind="farfield", nx=256, ny=256, nz=256, inset=10, nth=181, nph=361),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: any of the kinds, sizes spread over their logarithm."""
    kind = rng.choice(["solve", "solve", "solve", "batch", "farfield"])
    if kind == "batch":
        lo = rng.randint(36, 80)
        return dict(kind="batch", count=_log(rng, 3, 32), lo=lo, hi=lo + rng.randint(4, 80), tfsf=rng.choice([0.0, 0.3]),
                    steps=rng.randint(24, 64))
    if kind == "farfield":
        g = [_log(rng, 40, 220) for _ in range(3)]
        nth, nph = rng.choice([(61, 73), (181, 2), (37, 73), (91, 181)])
        return dict(kind="farfield", nx=g[0], ny=g[1], nz=g[2], inset=rng.randint(4, 12), nth=nth, nph=nph)
    form = rng.choice(["port", "graded", "unique", "tfsf", "dispersive"])
    steps = rng.randint(40, 100)
    if form == "port":
        return _drawn([_log(rng, 12, 200) for _ in range(3)], steps, mur=rng.choice(["none", "five", "six"]),
                      interval=rng.randint(1, 20))
    if form == "graded":
        return _drawn([_log(rng, 30, 110) for _ in range(3)], steps, coef="arrays", pml=rng.choice([6, 8]),
                      interval=rng.randint(1, 8))
    if form == "unique":
        return _drawn([_log(rng, 24, 120) for _ in range(3)], steps, coef="unique", mur=rng.choice(["five", "six"]),
                      interval=rng.randint(1, 8))
    if form == "tfsf":
        faces = rng.choice(["z", "all"])
        return _drawn([_log(rng, 64, 300) for _ in range(3)], steps, pml=8, faces=faces, mur="xy" if faces == "z" else "none",
                      source="tfsf", nfreq=rng.randint(1, 6), angle=rng.choice([0.0, 20.0, 45.0]))
    return _drawn([_log(rng, 64, 200) for _ in range(3)], steps, pml=8, source="tfsf", angle=30.0, nfreq=rng.randint(1, 5),
                  ade=rng.choice(["state", "apply"]))


def _drawn(grid, steps, **more):
    d = _solve("", grid, steps, **more)
    del d["name"]
    return d


# ---- inputs -------------------------------------------------------------------------------------------------------------

def _lines(case, axis):
    """Mesh lines of one axis: uniform, or graded at both ends; "unique" makes every spacing its own."""
    n = (case["nx"], case["ny"], case["nz"])[axis]
    if case["coef"] == "table":
        return opgen.uniform_lines(n, DELTA)
    d = np.full(n - 1, DELTA)
    end = max(1, n // 8)
    d[:end] *= np.minimum(1.2 ** np.arange(end, 0, -1), 2.0)
    d[-end:] *= np.minimum(1.2 ** np.arange(1, end + 1), 2.0)
    if case["coef"] == "unique":
        d *= 1.0 + 0.2 * np.sin(1.7 * np.arange(n - 1) + axis) * np.linspace(0.5, 1.0, n - 1)
    return np.concatenate([[0.0], np.cumsum(d)])


def _boxes(grid, W, faces):
    if faces == "z":
        return [((0, 0, 0), (grid[0], grid[1], W)), ((0, 0, grid[2] - W), (grid[0], grid[1], W))]
    Nx, Ny, Nz = grid
    return [((0, 0, 0), (W, Ny, Nz)), ((Nx - W, 0, 0), (W, Ny, Nz)),
            ((W, 0, 0), (Nx - 2 * W, W, Nz)), ((W, Ny - W, 0), (Nx - 2 * W, W, Nz)),
            ((W, W, 0), (Nx - 2 * W, Ny - 2 * W, W)), ((W, W, Nz - W), (Nx - 2 * W, Ny - 2 * W, W))]


_MUR = {"xy": [(0, "lo"), (0, "hi"), (1, "lo"), (1, "hi")],
        "five": [(0, "lo"), (0, "hi"), (1, "lo"), (1, "hi"), (2, "hi")],
        "six": [(a, s) for a in range(3) for s in ("lo", "hi")]}


def _insets(case):
    """(first cell of the region materials may fill, TFSF inset, NF2FF inset); smaller boxes on small grids."""
    small = min(case["nx"], case["ny"], case["nz"]) < 90
    nf, tf = (case["pml"] + 2, case["pml"] + 5) if small else (10, 20)
    return (tf + 3 if case["source"] == "tfsf" else max(case["pml"] + 2, 3)), tf, nf


@functools.lru_cache(maxsize=2)
def _fixed(key):
    """What the mesh alone decides, made once by a user's program: UPML, Mur, TFSF and NF2FF inputs, the vacuum rows."""
    case = dict(key)
    grid = (case["nx"], case["ny"], case["nz"])
    mesh = opgen.Mesh(*[_lines(case, a) for a in range(3)])
    dT = opgen.cfl_dt(mesh)
    W, f = case["pml"], {}
    wide = [W if case["faces"] == "all" or a == 2 else 0 for a in range(3)]
    sig = [opgen.pml_sigma(mesh, a, wide[a], wide[a]) if wide[a] else None for a in range(3)]
    if W:
        f["pml"] = opgen.upml_apply(mesh, dT, _boxes(grid, W, case["faces"]), sig, build=True)
    if case["mur"] != "none":
        f["mur"] = opgen.mur_dual(mesh, dT, _MUR[case["mur"]],
                                  ranges=[(wide[a], grid[a] - 1 - wide[a]) if wide[a] else None for a in range(3)])
    if case["coef"] == "table":
        # rows of a uniform mesh depend on the distance to each wall only: taken from a small mesh with the same ends
        e = [max(w, 1) for w in wide]
        R = [2 * w + 3 for w in e]
        m = opgen.Mesh(*[opgen.uniform_lines(r, DELTA) for r in R])
        arrs = opgen.operator_dense(m, dT)
        if W:
            opgen.upml_apply(m, dT, _boxes(R, W, case["faces"]),
                             [opgen.pml_sigma(m, a, wide[a], wide[a]) if wide[a] else None for a in range(3)], *arrs,
                             build=False)
        rows = np.concatenate([a.reshape(3, -1) for a in arrs]).T          # (cells of the small mesh, 12)
        r = []
        for a in range(3):
            i = np.full(grid[a], e[a] + 1)
            i[:e[a] + 1] = np.arange(e[a] + 1)
            i[grid[a] - e[a] - 1:] = np.arange(R[a] - e[a] - 1, R[a])
            r.append(i.astype(np.uint32))
        f["rows"] = rows
        f["mat"] = np.ascontiguousarray((r[0][:, None, None] * R[1] + r[1][None, :, None]) * R[2] + r[2][None, None, :], np.uint32)
        f["inner"] = int(((e[0] + 1) * R[1] + e[1] + 1) * R[2] + e[2] + 1)
    if case["source"] == "tfsf":
        row = f["rows"][f["inner"]]
        _, tf, nf = _insets(case)
        th = math.radians(case["angle"])
        vp, cp = opgen.tfsf_plane_wave(mesh, dT, [tf] * 3, [n - 1 - tf for n in grid], (math.sin(th), 0.0, math.cos(th)),
                                       (math.cos(th), 0.0, -math.sin(th)),
                                       lambda k, c, i: np.full(len(i), row[(3 if k == "E" else 9) + c]), 1 << 14)
        f["tfsf"] = dict(period=0, voltagePoints=vp, currentPoints=cp)
    if case["nfreq"]:
        f["surface"] = opgen.nf2ff_box(mesh, [nf] * 3, [n - 1 - nf for n in grid])
    return mesh, dT, sig, f


def _key(case):
    names = ("nx", "ny", "nz", "coef", "pml", "faces", "mur", "source", "angle", "nfreq")
    return tuple((k, case[k]) for k in names)


def _spheres(rng, grid, margin, cover):
    """Cells of seeded spheres, Drude and Lorentz, covering `cover` of the grid (at most half of what the margin leaves)."""
    label = np.zeros(grid, np.uint8)
    room = [n - 2 * margin for n in grid]
    target = min(cover * label.size, 0.4 * max(1, np.prod([max(0, r) for r in room])))
    rmax = max(1, min(40, min(room) // 2 - 1))
    done = 0
    for _ in range(4000):
        if done >= target:
            break
        r = int(rng.integers(max(1, rmax // 2), rmax + 1))
        c = [int(rng.integers(margin + r, max(margin + r + 1, n - margin - r))) for n in grid]
        sl = tuple(slice(v - r, v + r + 1) for v in c)
        ax = np.arange(-r, r + 1) ** 2
        ball = (ax[:, None, None] + ax[None, :, None] + ax[None, None, :]) <= r * r
        sub = label[sl]
        new = ball & (sub == 0)
        sub[new] = 1 + (rng.random() < 0.5)
        done += int(new.sum())
    return [np.flatnonzero(label.reshape(-1) == k).astype(np.uint32) for k in (1, 2)]


def _job(case, seed):
    """The engine inputs of one solve, in the form `workloads.configure` takes."""
    rng = np.random.default_rng(seed)
    grid = (case["nx"], case["ny"], case["nz"])
    mesh, dT, sig, f = _fixed(_key(case))
    job = dict(grid=list(grid), dT=dT, maxTS=max(4 * case["steps"], 400), endCrit=0.0)
    lo, _, _ = _insets(case)
    boxes = []
    for i in range(12):
        size = [int(rng.integers(1, max(2, n // 6))) for n in grid]
        a = [int(rng.integers(min(lo, n - 1), max(min(lo, n - 1) + 1, n - lo - s))) for n, s in zip(grid, size)]
        boxes.append(tuple(slice(p, min(p + s, max(n - lo, p + 1))) for p, s, n in zip(a, size, grid)))
    eps = rng.uniform(2.0, 10.0, 12)
    if case["coef"] == "table":
        mat, inner = f["mat"].copy(), f["rows"][f["inner"]]
        rows = [f["rows"]]
        for i, b in enumerate(boxes):          # dielectric, lossy dielectric, metal in turn
            row, a = inner.copy(), 0.002 * (i % 3 == 1)
            row[:3] = (1 - a) / (1 + a) if i % 3 < 2 else 0.0
            row[3:6] = inner[3:6] / eps[i] / (1 + a) if i % 3 < 2 else 0.0
            mat[b] = len(f["rows"]) + i
            rows.append(row[None])
        if case["ade"] != "none":
            cells = _spheres(rng, grid, lo, 0.3)
            dr = [opgen.ade_drude(inner[n:n + 1], inner[3 + n:4 + n], dT, 1.4e16, 3e13) for n in range(3)]
            lz = [opgen.ade_lorentz(inner[n:n + 1], inner[3 + n:4 + n], dT, 2.0, 2 * math.pi * 15e9, 2 * math.pi * 1e9)
                  for n in range(3)]
            base = sum(len(r) for r in rows)
            flat = mat.reshape(-1)
            for k in range(2):
                row = inner.copy()
                if k == 0 and case["ade"] == "apply":       # the stiff metal's implicit scheme has its own row
                    for n in range(3):
                        row[n], row[3 + n] = dr[n]["vv"][0], dr[n]["vi"][0]
                flat[cells[k]] = base + k
                rows.append(row[None])
            orders = []
            for k, co in ((0, dr), (1, lz)):
                m = len(cells[k])
                full = lambda v: np.full(m, v, np.float32)  # noqa: E731
                orders.append(dict(numCells=m, hasLorentz=bool(k), directions=[
                    dict(dir=n, pos_idx=cells[k], v_int_ADE=full(co[n]["v_int"][0]), v_ext_ADE=full(co[n]["v_ext"][0]),
                         **({"v_Lor_ADE": full(co[n]["v_lor"][0])} if k else {})) for n in range(3)]))
            job["ade"] = dict(orders=orders, apply=case["ade"] == "apply")
        job["coefficients"] = dict(mat=mat.reshape(-1), table=np.concatenate(rows).astype(np.float32))
    else:
        e = np.ones([n - 1 for n in grid])
        kap = np.zeros([n - 1 for n in grid])
        for i, b in enumerate(boxes):
            e[b] = eps[i]
            kap[b] = 0.02 * (i % 3 == 1)
        arrs = opgen.operator_dense(mesh, dT, eps_r=e, kappa=kap)
        if case["pml"]:
            opgen.upml_apply(mesh, dT, _boxes(grid, case["pml"], case["faces"]), sig, *arrs, build=False)
        job["coefficients"] = dict(zip(("vv", "vi", "ii", "iv"), (opgen.flat(a) for a in arrs)))
    if "pml" in f:
        job["pml"] = f["pml"]
    if "mur" in f:
        job["mur"] = f["mur"]
    pulse = (rng.uniform(0.5, 2.0) * opgen.gauss_signal(F0, rng.uniform(0.6, 1.0) * FC, dT)).astype(np.float32)
    if case["source"] == "tfsf":
        job["tfsf"] = dict(f["tfsf"], signal=pulse)
    else:
        x, y, z = (n // 2 for n in grid)
        k = min(3, grid[2] - 1 - z)
        at = (x * grid[1] + y) * grid[2] + z
        job["excitation"] = dict(signal=pulse, delay=[0] * k, amp=[1.0 / k] * k, dir=[2] * k, pos=[at + i for i in range(k)],
                                 period=0)
        job["probes"] = [opgen.voltage_probe(mesh, (x, y, z), (x, y, z + k), interval=case["interval"]),
                         opgen.current_probe(mesh, (x - 1, y - 1, z), (x, y, z), 2, interval=case["interval"])]
    if case["nfreq"]:
        pts, meta, primal, dual = f["surface"]
        job["nf2ff"] = dict(surfaceIndices=pts.ravel(), numPoints=len(pts), dT=dT, gridSize=list(grid), primalEdgeLens=primal,
                            dualEdgeLens=dual, maxTS=job["maxTS"], windowType=0,
                            omegas=[2 * math.pi * (F0 + FC * (k / max(1, case["nfreq"] - 1) - 0.5)) for k in range(case["nfreq"])])
        job["meta"] = meta
    return job


def _start_fields(case, seed):
    """E and H of a solve under way, (3, Nx, Ny*Nz): volts of order 1, currents of order 1/Z0."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    shape = (3, case["nx"], case["ny"] * case["nz"])
    return torch.randn(shape, device="cuda", generator=g), torch.randn(shape, device="cuda", generator=g) / Z0


def _members(case, seed):
    """The solves of a batch: sizes as the sweep's (fixed by the case), every member with a seed of its own."""
    rng = np.random.default_rng(case["count"] * 1000 + case["lo"])
    out = []
    for i in range(case["count"]):
        g = [int(v) for v in rng.integers(case["lo"], case["hi"] + 1, 3)]
        wave = i < round(case["tfsf"] * case["count"])
        out.append((_drawn(g, case["steps"], source="tfsf" if wave else "port", nfreq=2 if wave else 0, mur="six" if wave else "five",
                           interval=13), seed * 1000 + i))
    return out


def _far_case(case):
    c = dict(BASE, nx=case["nx"], ny=case["ny"], nz=case["nz"], steps=16)
    return c


def _far_job(case, seed):
    c = _far_case(case)
    job = _job(c, seed)
    mesh, dT, _, _ = _fixed(_key(c))
    grid = (c["nx"], c["ny"], c["nz"])
    pts, meta, primal, dual = opgen.nf2ff_box(mesh, [case["inset"]] * 3, [n - 1 - case["inset"] for n in grid])
    job["nf2ff"] = dict(surfaceIndices=pts.ravel(), numPoints=len(pts), dT=dT, gridSize=list(grid), primalEdgeLens=primal,
                        dualEdgeLens=dual, maxTS=100, windowType=0, omegas=[2 * math.pi * F0])
    job["meta"] = meta
    job["theta"] = np.linspace(0.0, math.pi, case["nth"]).astype(np.float32)
    job["phi"] = np.linspace(0.0, 2 * math.pi, case["nph"]).astype(np.float32)
    job["center"] = [float(0.5 * DELTA * (n - 1)) for n in grid]
    return c, job


# ---- the calls ----------------------------------------------------------------------------------------------------------

def _engine(case, job, seed):
    e = CudaEngine()
    if not e.initGPU():
        raise RuntimeError("no CUDA device")
    workloads.configure(e, job)
    volt, curr = _start_fields(case, seed)
    torch.cuda.synchronize()
    e.setPlanes(0, volt, curr)
    return e


def _room(cells):
    return torch.empty(3 * cells, device="cuda"), torch.empty(3 * cells, device="cuda")


def prepare(case, seed):
    if case["kind"] == "farfield":
        c, job = _far_job(case, seed)
        e = _engine(c, job, seed)
        e.iterate(16)
        e.sync()
        return dict(kind="farfield", engine=e, config=dict(
            pointMeta=job["meta"], theta=job["theta"], phi=job["phi"], center=job["center"], frequency=F0, radius=1.0,
            numPoints=job["nf2ff"]["numPoints"], freqIndex=0))
    if case["kind"] == "batch":
        engines, cells = [], 0
        for c, s in _members(case, seed):
            engines.append(_engine(c, _job(c, s), s))
            cells += engines[-1].totalCells
        E, H = _room(cells)
        views, at = [], 0
        for e in engines:
            n = 3 * e.totalCells
            shape = (3, e.numLines[0], e.numLines[1] * e.numLines[2])
            views.append((E[at:at + n].view(shape), H[at:at + n].view(shape)))
            at += n
        return dict(kind="batch", engines=engines, batch=CudaBatch(engines), steps=case["steps"], E=E, H=H, views=views)
    e = _engine(case, _job(case, seed), seed)
    E, H = _room(e.totalCells)
    shape = (3, case["nx"], case["ny"] * case["nz"])
    return dict(kind="solve", engine=e, steps=case["steps"], E=E.view(shape), H=H.view(shape), nf=case["nfreq"] > 0)


def run(state):
    if state["kind"] == "farfield":
        return state["engine"].computeNF2FFfarField(state["config"])
    if state["kind"] == "batch":
        state["batch"].iterate(state["steps"])
        rings, acc = [], []
        for e, (E, H) in zip(state["engines"], state["views"]):
            r = e.readProbeGatherBuffered()
            if r is not None:
                rings.append(r["data"])
            a = e.readNF2FFAccumulation(True)
            if a is not None:
                acc += [a["accumE"].ravel(), a["accumH"].ravel()]
            e.getPlanes(0, e.numLines[0], out=(E, H))
        out = dict(E=state["E"], H=state["H"])
        if rings:
            out["rings"] = np.concatenate(rings)
        if acc:
            out["acc"] = np.concatenate(acc)
        return out
    e = state["engine"]
    e.iterate(state["steps"])
    out = dict(energy=e.computeEnergy(lagged=False))
    ring = e.readProbeGatherBuffered()
    if ring is not None:
        out["ring"] = ring["data"]
    if state["nf"]:
        out.update(e.readNF2FFAccumulation(True))
    out["E"], out["H"] = e.getPlanes(0, e.numLines[0], out=(state["E"], state["H"]))
    return out


# ---- what a pass cannot do without --------------------------------------------------------------------------------------

def _step_bytes(case):
    """Bytes and operations of one timestep: every field value read and written once, a coefficient tuple (or its index)
    per cell, the UPML fluxes, the Mur pairs, the ADE state, the NF2FF samples."""
    n = case["nx"] * case["ny"] * case["nz"]
    b = n * (48 + (48 if case["coef"] == "unique" else 4))
    grid = (case["nx"], case["ny"], case["nz"])
    u = 0
    if case["pml"]:
        u = sum(p[0] * p[1] * p[2] for _, p in _boxes(grid, case["pml"], case["faces"]))
    b += u * 50
    if case["mur"] != "none":
        b += 12 * sum(2 * n // grid[a] for a, _ in _MUR[case["mur"]])
    if case["ade"] != "none":
        margin, _, _ = _insets(case)
        ent = 3 * min(0.3 * n, 0.4 * max(0, math.prod(g - 2 * margin for g in grid)))
        b += int(ent * 12)
    if case["nfreq"]:
        _, _, nf = _insets(case)
        s = [g - 2 * nf for g in grid]
        b += 2 * (s[0] * s[1] + s[1] * s[2] + s[0] * s[2]) * 24
    return b, n * 42 + u * 24


def work(case):
    if case["kind"] == "farfield":
        s = [n - 2 * case["inset"] for n in (case["nx"], case["ny"], case["nz"])]
        pts = 2 * (s[0] * s[1] + s[1] * s[2] + s[0] * s[2])
        return {"bytes": pts * 80 + case["nth"] * case["nph"] * 20, "flops": 40.0 * pts * case["nth"] * case["nph"]}
    if case["kind"] == "batch":
        w = [_step_bytes(c) for c, _ in _members(case, 0)]
        return {"bytes": case["steps"] * sum(x[0] for x in w), "flops": case["steps"] * sum(x[1] for x in w)}
    b, f = _step_bytes(case)
    return {"bytes": case["steps"] * b, "flops": case["steps"] * f}


# ---- the same in 64 bits ------------------------------------------------------------------------------------------------

def _dev(a, dtype=torch.float64):
    a = np.asarray(a)
    return torch.as_tensor(a.astype(np.int64) if a.dtype == np.uint32 else a, device="cuda").to(dtype)


def _last(idx):
    """(distinct targets, the last entry that writes each)."""
    rev = np.asarray(idx)[::-1]
    t, first = np.unique(rev, return_index=True)
    return t, len(rev) - 1 - first


class _Exact:
    """The reference's timestep (phase order of CPUFDTDEngine.step, webgpu-fdtd.mjs:1129-1172) on f64 tensors."""

    def __init__(self, case, job, seed):
        g = self.g = tuple(job["grid"])
        shape = (3,) + g
        volt, curr = _start_fields(case, seed)
        self.E, self.H = volt.double().view(shape), curr.double().view(shape)
        c = job["coefficients"]
        if "mat" in c:
            m, t = _dev(c["mat"], torch.int64).int(), _dev(c["table"])
            self.k = [torch.stack([torch.index_select(t[:, 3 * a + n], 0, m).view(g) for n in range(3)]) for a in range(4)]
        else:
            self.k = [_dev(c[n]).view(shape) for n in ("vv", "vi", "ii", "iv")]
        self.pml = []
        for r in job.get("pml") or []:
            sl = (slice(None),) + tuple(slice(a, a + b) for a, b in zip(r["startPos"], r["numLines"]))
            s3 = (3,) + tuple(r["numLines"])
            co = {n: _dev(r[n]).view(s3) for n in ("vv", "vvfo", "vvfn", "ii", "iifo", "iifn")}
            self.pml.append((sl, co, torch.zeros(s3, dtype=torch.float64, device="cuda"),
                             torch.zeros(s3, dtype=torch.float64, device="cuda")))
        self.job, self.n = job, 0
        m = job.get("mur")
        if m:
            cat = lambda k: np.concatenate([m[k + "_nyP"], m[k + "_nyPP"]])  # noqa: E731
            nrm = cat("normal_idx")
            t, last = _last(nrm)
            self.mur = [_dev(cat("coeff")), _dev(nrm, torch.int64), _dev(cat("shifted_idx"), torch.int64),
                        _dev(t, torch.int64), _dev(last, torch.int64)]
        self.ade = []
        for o in (job.get("ade") or {}).get("orders", []):
            for d in o["directions"]:
                if o["numCells"]:
                    at = _dev(d["pos_idx"], torch.int64) + d["dir"] * math.prod(g)
                    z = torch.zeros(len(at), dtype=torch.float64, device="cuda")
                    self.ade.append([at, float(d["v_int_ADE"][0]), float(d["v_ext_ADE"][0]),
                                     float(d["v_Lor_ADE"][0]) if o["hasLorentz"] else None, z, z.clone()])
        if job.get("tfsf"):
            f = job["tfsf"]
            self.sig = _dev(f["signal"])
            self.tf = [[_dev(p["field_idx"], torch.int64), _dev(p["delay_int"], torch.int64), _dev(p["delay_frac"]), _dev(p["amp"])]
                       for p in (f["voltagePoints"], f["currentPoints"])]
        if job.get("nf2ff"):
            f = job["nf2ff"]
            self.pts = _dev(f["surfaceIndices"], torch.int64).view(-1, 3)
            self.pl = [_dev(a) for a in f["primalEdgeLens"]]
            self.dl = [_dev(a) for a in f["dualEdgeLens"]]
            self.acc = torch.zeros((2, len(f["omegas"]), f["numPoints"], 3, 2), dtype=torch.float64, device="cuda")
        self.ring = []
        self.probe = None
        if job.get("probes"):
            idx, _ = opgen.build_gather_indices(job["probes"], g)
            self.probe = _dev(idx, torch.int64)

    def points(self, F, side):
        if not self.job.get("tfsf"):
            return
        at, delay, frac, amp = self.tf[side]
        d = self.n - delay
        ok = (d >= 0) & (d < len(self.sig) - 1)
        d = d.clamp(0, len(self.sig) - 2)
        v = amp * ((1 - frac) * self.sig[d] + frac * self.sig[d + 1])
        F.view(-1).index_add_(0, at, torch.where(ok, v, torch.zeros_like(v)))

    def half(self, F, a, names, curl):
        help_ = []
        for sl, co, *flux in self.pml:
            fo = flux[a]
            help_.append(co[names[0]] * F[sl] - co[names[1]] * fo)
            F[sl] = fo
        yield
        curl()
        for (sl, co, *flux), h in zip(self.pml, help_):
            flux[a].copy_(F[sl])
            F[sl] = h + co[names[2]] * flux[a]

    def curl_e(self):
        E, H, (vv, vi) = self.E, self.H, self.k[:2]
        for n in range(3):
            p, q = (n + 1) % 3, (n + 2) % 3
            c = self.back(H[q], p) - self.back(H[p], q)
            E[n].mul_(vv[n]).add_(c.mul_(vi[n]))

    def curl_h(self):
        E, H, (ii, iv) = self.E, self.H, self.k[2:]
        s = tuple(slice(0, n - 1) for n in self.g)
        for n in range(3):
            p, q = (n + 1) % 3, (n + 2) % 3
            c = -E[q].diff(dim=p)[s] + E[p].diff(dim=q)[s]
            H[n][s] = H[n][s] * ii[n][s] + c.mul_(iv[n][s])

    @staticmethod
    def back(a, dim):
        """a - a(-1) along dim; index 0 refers to itself."""
        out = torch.zeros_like(a)
        out.narrow(dim, 1, a.shape[dim] - 1).copy_(a.diff(dim=dim))
        return out

    def step(self):
        E, H = self.E, self.H
        e = self.half(E, 0, ("vv", "vvfo", "vvfn"), self.curl_e)
        next(e)
        for s in self.ade:
            at, kint, kext, klor, st, lor = s
            v = E.view(-1)[at]
            if klor is not None:
                lor.add_(klor * st)
                v = v - lor
            st.mul_(kint).add_(kext * v)
        if self.job.get("mur"):
            c, nrm, shf, t, last = self.mur
            saved = E.view(-1)[shf] - c * E.view(-1)[nrm]
        next(e, None)
        self.points(E, 0)
        if self.job.get("mur"):
            saved += c * E.view(-1)[shf]
        x = self.job.get("excitation")
        if x:
            d = self.n if self.n < len(x["signal"]) else 0
            for amp, n, pos in zip(x["amp"], x["dir"], x["pos"]):
                E[n].view(-1)[pos] += float(np.float32(amp)) * float(x["signal"][d])
        if self.job.get("mur"):
            E.view(-1)[t] = saved[last]
        if (self.job.get("ade") or {}).get("apply"):
            for s in self.ade:
                E.view(-1)[s[0]] -= s[4]
        h = self.half(H, 1, ("ii", "iifo", "iifn"), self.curl_h)
        next(h)
        next(h, None)
        self.points(H, 1)
        self.n += 1
        if self.job.get("nf2ff"):
            self.sample()
        if self.probe is not None and self.n % self.job["probes"][0]["processInterval"] == 0:
            self.ring.append(torch.stack([E.view(-1)[self.probe], H.view(-1)[self.probe]], dim=1).reshape(-1))

    def sample(self):
        f, P, N, g = self.job["nf2ff"], self.pts, math.prod(self.g), self.g
        st = (g[1] * g[2], g[2], 1)
        base = P[:, 0] * st[0] + P[:, 1] * st[1] + P[:, 2]
        Ef, Hf, f64 = self.E.view(-1), self.H.view(-1), torch.float64
        for n in range(3):
            p, q = (n + 1) % 3, (n + 2) % 3
            b = n * N + base
            e = (Ef[b] + Ef[b + st[p]] + Ef[b + st[q]] + Ef[b + st[p] + st[q]]) / (4 * self.pl[n][P[:, n]])
            d0, d1 = self.dl[n][P[:, n]], self.dl[n][P[:, n] + 1]
            r = d0 / (d0 + d1)
            h = Hf[b] / d0 * (1 - r) + Hf[b + st[n]] / d1 * r
            for k, w in enumerate(f["omegas"]):
                for a, (v, t) in enumerate(((e, self.n), (h, self.n + 0.5))):
                    ph = w * f["dT"] * t
                    wt = float(np.float32(f["dT"]))
                    self.acc[a, k, :, n] += v[:, None] * torch.tensor([math.cos(ph) * wt, -math.sin(ph) * wt], dtype=f64, device="cuda")

    def energy(self):
        s = (slice(None),) + tuple(slice(0, n - 1) for n in self.g)
        return float(self.E[s].square().sum() + self.H[s].square().sum())


def _far_exact(case, x, job):
    """N and L sums over the surface points (webgpu-engine.mjs:830-985), as one complex product per block of angles."""
    meta = _dev(job["meta"])
    pos = meta[:, :3] - _dev(job["center"])
    nd, s = meta[:, 3].long(), meta[:, 4] * meta[:, 5]
    E, H = (torch.view_as_complex(x.acc[a, 0].contiguous()) for a in range(2))
    i = torch.arange(len(nd), device="cuda")
    cur = torch.zeros((len(nd), 6), dtype=torch.complex128, device="cuda")
    a, b = (nd + 1) % 3, (nd + 2) % 3
    cur[i, a], cur[i, b] = -s * H[i, b], s * H[i, a]
    cur[i, 3 + a], cur[i, 3 + b] = s * E[i, b], -s * E[i, a]
    th, ph = _dev(job["theta"]), _dev(job["phi"])
    T, Q = (v.reshape(-1) for v in torch.meshgrid(th, ph, indexing="ij"))
    u = torch.stack([T.sin() * Q.cos(), T.sin() * Q.sin(), T.cos()], dim=1)
    k = 2 * math.pi * F0 / C0
    NL = torch.empty((len(T), 6), dtype=torch.complex128, device="cuda")
    for j in range(0, len(T), 512):
        arg = k * (u[j:j + 512] @ pos.T)
        NL[j:j + 512] = torch.polar(torch.ones_like(arg), arg) @ cur
    pt = lambda v: v[:, 0] * T.cos() * Q.cos() + v[:, 1] * T.cos() * Q.sin() - v[:, 2] * T.sin()  # noqa: E731
    pp = lambda v: v[:, 1] * Q.cos() - v[:, 0] * Q.sin()  # noqa: E731
    N, L = NL[:, :3], NL[:, 3:]
    fac = k / (4 * math.pi) * complex(math.sin(k), math.cos(k))        # j k e^{-jk r} / (4 pi r), r = 1
    Et, Ep = -fac * (pp(L) + Z0 * pt(N)), fac * (pt(L) - Z0 * pp(N))
    P = (Et.abs() ** 2 + Ep.abs() ** 2) / (2 * Z0)
    return torch.stack([P, Et.real, Et.imag, Ep.real, Ep.imag], dim=1).reshape(-1)


def _solve_exact(case, seed):
    job = _job(case, seed)
    x = _Exact(case, job, seed)
    for _ in range(case["steps"]):
        x.step()
    return x


def exact(case, seed):
    if case["kind"] == "farfield":
        c, job = _far_job(case, seed)
        x = _Exact(c, job, seed)
        for _ in range(16):
            x.step()
        return _far_exact(case, x, job).cpu().numpy()
    if case["kind"] == "batch":
        E, H, rings, acc = [], [], [], []
        for c, s in _members(case, seed):
            x = _solve_exact(c, s)
            E.append(x.E.reshape(-1))
            H.append(x.H.reshape(-1))
            rings += x.ring
            if c["nfreq"]:
                acc += [x.acc[0].reshape(-1), x.acc[1].reshape(-1)]
        out = dict(E=torch.cat(E), H=torch.cat(H))
        if rings:
            out["rings"] = torch.cat(rings).cpu().numpy()
        if acc:
            out["acc"] = torch.cat(acc).cpu().numpy()
        return out
    x = _solve_exact(case, seed)
    shape = (3, case["nx"], case["ny"] * case["nz"])
    out = dict(energy=x.energy(), E=x.E.view(shape), H=x.H.view(shape))
    if x.ring:
        out["ring"] = torch.cat(x.ring).cpu().numpy()
    if case["nfreq"]:
        for a, name in enumerate(("accumE", "accumH")):
            out[name] = x.acc[a].reshape(case["nfreq"], -1).cpu().numpy()
    return out
