"""The calls that users of this framework wait for, as measurable cases.

A case is a dict of plain values: the shape of a specimen (a seeded bcc tip in
its vacuum box, Mesh.from_tip), the kind of call, and that call's size and
options.  prepare() makes what a program has in hand before the call (the
device grid of a specimen from which a few seeded surface atoms have gone
already, relaxed; the plan and options it keeps; the ions it will launch),
run() makes one pass through the public entry points.

    event     Evaporation.step / Evaporation.run: whole evaporation events
    trace     Grid.trace: a batch of probe ions on a relaxed specimen
    relax     Grid.solve from a cold start to a relative residual, and the
              potentials and fields it leaves (the relaxation command)
    sweep     Grid.relax: the reference's coloured sweeps over the free cells
    snapshot  the values of the grid and surface logs after an event
    tips      serving.run_tips: one event on each of several specimens
    train     Learner.train: Adam steps of the learned warm start's network
"""
from __future__ import annotations

import math

import numpy as np
import torch

from tapsim_modified_b200 import serving
from tapsim_modified_b200.tapsim import Evaporation, EvaporationOptions, Grid, Learner, Mesh, solve_opts

VACUUM = 0
# atoms gone from the surface before the first measured call
GONE = 12
# relative residual of the events' relaxations, the value the headline runs at
REL_TOL = 1e-8
# and of a specimen's own relaxation from a cold start, whose far field is
# still 1e-4 off at 1e-8
COLD_TOL = 1e-10
# the 1 um box of the documented tips
BOX = dict(box_half_width=0.5e-6, box_height=1.0e-6, fine_shell=3e-9)
# config-1 tip: 5 nm cap on a 10 nm cylinder, 307k cells
TIP5 = dict(cap_radius=5e-9, shank_length=10e-9, half_angle_deg=0.0, solute_fraction=0.0, **BOX)
# the larger end: 835k cells
MID = dict(cap_radius=8e-9, shank_length=15e-9, half_angle_deg=5.0, solute_fraction=0.0, **BOX)
# small specimen in a small box: 23k cells
SMALL = dict(cap_radius=2e-9, shank_length=4e-9, half_angle_deg=0.0, solute_fraction=0.0,
             box_half_width=50e-9, box_height=200e-9, fine_shell=0.8e-9)
# Fe-1.5 at.% Cu with precipitates, the probe-ion specimen at a smaller cap
ALLOY = dict(cap_radius=6e-9, shank_length=15e-9, half_angle_deg=0.0, solute_fraction=0.015, **BOX)
PRECIPITATES = dict(precip_density=2e24, precip_rmin=1e-9, precip_rmax=2e-9)
SHAPE = ("cap_radius", "shank_length", "half_angle_deg", "solute_fraction", "box_half_width", "box_height",
         "fine_shell")


def listed():
    return [
        # the smallest call: one event on a small specimen, as an interactive
        # run or a parameter study makes them; launches and latency count
        dict(name="event_small", kind="event", count=1, warm_start=0, relax_mode=1, tip_seed=3, **SMALL),
        # one event at a time on the config-1 tip (a program that looks at
        # each record before the next event)
        dict(name="event_tip5", kind="event", count=1, warm_start=0, relax_mode=1, tip_seed=11, **TIP5),
        # the ordinary run: events in batches, flights beside the next events
        dict(name="events_tip5", kind="event", count=16, warm_start=0, relax_mode=1, tip_seed=11, **TIP5),
        # the same on the larger specimen, from the recycled correction
        dict(name="events_mid", kind="event", count=8, warm_start=1, relax_mode=1, tip_seed=5, **MID),
        # the drop-in run with the shipped tapsim.ini: local relaxation and a
        # global sweep per event
        dict(name="events_default_ini", kind="event", count=4, warm_start=0, relax_mode=0, tip_seed=11, **TIP5),
        # 4096 probe ions per event, FP64 flights (hit maps)
        dict(name="probe_fp64", kind="trace", ions=4096, precision=0, tip_seed=2, **ALLOY),
        # fewer ions, FP64 near the tip and FP32 beyond
        dict(name="probe_mixed", kind="trace", ions=500, precision=2, tip_seed=11, **TIP5),
        # the relaxation command on the larger specimen
        dict(name="relax_mid", kind="relax", tip_seed=5, **MID),
        # the reference's own relaxation: 25 sweeps over all free cells
        dict(name="sweep_tip5", kind="sweep", cycles=25, tip_seed=11, **TIP5),
        # grid and surface logs of an alloy specimen
        dict(name="snapshot_alloy", kind="snapshot", tip_seed=2, **ALLOY),
        # many-tip serving: one event on each of six specimens
        dict(name="tips_6", kind="tips", tips=6, warm_start=1, tip_seed=21,
             **dict(TIP5, cap_radius=4e-9)),
        # training of the learned warm start: eight Adam steps of batch 8
        dict(name="train", kind="train", steps=8, batch=8, samples=24, tip_seed=3, **SMALL),
    ]


def draw(rng):
    """One more case of the same ranges: caps of 2 to 7.5 nm on shanks of 1.5
    to 2.5 cap radii, the counts between the smallest and largest listed."""
    cap = 2e-9 * 3.75 ** rng.random()
    small = cap < 3e-9
    c = dict(cap_radius=cap, shank_length=cap * rng.uniform(1.5, 2.2), half_angle_deg=rng.uniform(0.0, 4.0),
             solute_fraction=rng.choice([0.0, 0.015]), box_half_width=50e-9 if small else 0.5e-6,
             box_height=200e-9 if small else 1.0e-6, fine_shell=0.8e-9 if small else rng.uniform(2e-9, 3e-9),
             tip_seed=rng.randrange(1, 1000))
    kind = rng.choice(["event", "event", "event", "trace", "trace", "relax", "sweep", "snapshot", "tips", "train"])
    c["kind"] = kind
    if kind == "event":
        mode = rng.choice([1, 1, 1, 0])
        c.update(count=rng.choice([1, 1, 3, 7, 13, 16]) if mode == 1 else rng.randrange(1, 5),
                 warm_start=rng.choice([0, 1]) if mode == 1 else 0, relax_mode=mode)
    elif kind == "trace":
        c.update(ions=int(4096 ** rng.uniform(0.0, 1.0)), precision=rng.choice([0, 0, 2]))
    elif kind == "sweep":
        c.update(cycles=rng.randrange(1, 30))
    elif kind == "tips":
        c.update(tips=rng.randrange(2, 7), warm_start=rng.choice([0, 1]), cap_radius=min(cap, 4e-9),
                 shank_length=min(c["shank_length"], 10e-9))
    elif kind == "train":
        c.update(steps=rng.randrange(2, 12), batch=rng.randrange(2, 9), samples=24, cap_radius=min(cap, 3e-9),
                 shank_length=min(c["shank_length"], 6e-9))
    return c


# ---- specimens ------------------------------------------------------------

_meshes: dict = {}


def _mesh(case, k=0):
    """The host mesh of the case's k-th specimen and its arrays.  A program
    builds it once per specimen (seconds of host work) and keeps it; the last
    few are kept here."""
    key = tuple(case[f] for f in SHAPE) + (case["tip_seed"] + k,)
    if key not in _meshes:
        while len(_meshes) >= 16:
            _meshes.pop(next(iter(_meshes)))
        kw = {f: case[f] for f in SHAPE}
        if case["solute_fraction"] > 0.0:
            kw.update(PRECIPITATES)
        m = Mesh.from_tip(seed=key[-1], **kw)
        _meshes[key] = (m, m.arrays())
    return _meshes[key]


def _gone(a, seed):
    """The seeded surface atoms that have left the specimen already, no two
    of them in one neighbourhood."""
    row = np.repeat(np.arange(len(a["type"])), np.diff(a["row_ptr"]))
    removable = np.isin(a["type"], [t for t, v in a["types"].items() if v["removable"]])
    edge = removable[row] & (a["type"][a["col"]] == VACUUM) & (a["area_pos"] > 0)
    surface = np.unique(row[edge])
    out, taken = [], set()
    for i in np.random.default_rng(seed).permutation(surface):
        nb = a["col"][a["row_ptr"][i]:a["row_ptr"][i + 1]]
        if taken.isdisjoint(nb) and i not in taken:
            out.append(int(i))
            taken.add(int(i))
            taken.update(int(j) for j in nb)
        if len(out) == GONE:
            break
    return out


def _specimen(case, seed, k=0, relax=True):
    mesh, a = _mesh(case, k)
    g = Grid(mesh)
    g.surface_init(VACUUM)
    for node in _gone(a, seed + 7919 * k):
        g.take_away(node)
    if relax:
        g.solve(COLD_TOL, 50, 50000, 1e-4, preconditioner=1)
    return g, a


def _solve(warm_start):
    return solve_opts(rel_tol=REL_TOL, max_outer=50, max_inner=20000, warm_start=warm_start, preconditioner=1)


def _options():
    return EvaporationOptions.from_ini(None)


# ---- the cases ------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    s = dict(kind=kind, case=case)
    if kind == "event":
        s["grid"], _ = _specimen(case, seed)
        s["ev"] = Evaporation(s["grid"], _options(), relax_mode=case["relax_mode"], solve=_solve(case["warm_start"]))
    elif kind == "trace":
        g, a = _specimen(case, seed)
        s["grid"] = g
        cells, _ = g.surface()
        rng = np.random.default_rng(seed)
        pick = rng.choice(cells, size=case["ions"], replace=len(cells) < case["ions"])
        # ordered by azimuth and height, as the probe-ion runs order them
        xyz = a["xyz"][pick]
        order = np.lexsort((np.round(xyz[:, 2] / 1e-9), np.arctan2(xyz[:, 1], xyz[:, 0])))
        pick = pick[order]
        t = a["types"]
        q = {k: v["evap_charge"] * 1.60217733e-19 / (v["mass"] * 1.660538782e-27) for k, v in t.items()
             if v["mass"] > 0.0}
        s["start"] = a["xyz"][pick]
        s["qm"] = np.array([q[int(k)] for k in a["type"][pick]], np.float32)
        s["tet"] = a["node_tet"][pick]
        s["opts"] = dict(precision=case["precision"], fp64_radius=3.0 * case["cap_radius"])
    elif kind == "relax":
        s["grid"], a = _specimen(case, seed, relax=False)
        s["phi"] = _start(a, seed)
        # the program's first relaxation sets the hierarchy up, once per grid
        s["grid"].solve(0.5, 50, 50000, 1e-1, preconditioner=1)
    elif kind == "sweep":
        s["grid"], _ = _specimen(case, seed, relax=False)
    elif kind == "snapshot":
        s["grid"], _ = _specimen(case, seed)
    elif kind == "tips":
        s["grids"] = [_specimen(case, seed, k)[0] for k in range(case["tips"])]
        for g in s["grids"]:
            g.select()
        s["opts"] = [_options().event_opts(VACUUM, 1, _solve(case["warm_start"])) for _ in s["grids"]]
        s["index"] = 0
    elif kind == "train":
        g, _ = _specimen(case, seed)
        s["learner"] = Learner(hops=6, max_cells=1024, ell_width=64, seed=seed)
        s["learner"].attach(g, collect=True)
        Evaporation(g, _options(), relax_mode=1, solve=_solve(1), trace=False).run(case["samples"])
        s["learner"].attach(g)
        s["seed"] = seed
    return s


def _start(a, seed):
    """A cold start: the specimen at a seeded voltage, the rest as the mesh
    file has it."""
    return a["phi"].astype(np.float64) * np.random.default_rng(seed).uniform(0.5, 2.0)


def _rows(records):
    """The columns of the results file (LogResults::Dataset)."""
    f = np.float32
    return dict(node=np.array([r["node"] for r in records], np.int64),
                id=np.array([r["id"] for r in records], np.int64),
                voltage=np.array([r["voltage"] for r in records], f),
                stop=np.array([r["stop"] for r in records], f),
                tof=np.array([r["tof"] for r in records], f),
                probability=np.array([r["probability"] for r in records], f),
                potential_before=np.array([r["potentialBefore"] for r in records], f),
                field_before=np.array([r["fieldBefore"] for r in records], f),
                potential_after=np.array([r["potentialAfter"] for r in records], f),
                field_after=np.array([r["fieldAfter"] for r in records], f),
                normal=np.array([r["normal"] for r in records], f),
                apex=np.array([r["apex"] for r in records], f))


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "event":
        return _rows([s["ev"].step()] if case["count"] == 1 else s["ev"].run(case["count"]))
    if kind == "trace":
        imp = np.ctypeslib.as_array(s["grid"].trace(s["start"], s["qm"], s["tet"], **s["opts"]))
        return dict(stop=imp["stop"], stop_time=imp["stop_time"], status=imp["status"])
    if kind == "relax":
        g = s["grid"]
        g.set_potentials(s["phi"])
        g.solve(COLD_TOL, 50, 50000, 1e-4, preconditioner=1)
        phi, field, _ = g.cell_values(force=False)
        return dict(phi=phi, field=field)
    if kind == "sweep":
        dev = s["grid"].relax(case["cycles"])
        return dict(deviation=dev, phi=s["grid"].potentials())
    if kind == "snapshot":
        g = s["grid"]
        phi, field, force = g.cell_values()
        cells, prob = g.surface_cells()
        # the surface log's columns, by cell
        probability, normal = np.zeros(g.n, np.float32), np.zeros((g.n, 3), np.float32)
        probability[cells] = prob
        normal[cells] = g.surface_normals(cells)
        return dict(phi=phi, field=field, force=force, types=g.types(), probability=probability, normal=normal)
    if kind == "tips":
        s["index"] += 1
        recs, _, _ = serving.run_tips(s["grids"], s["opts"], s["index"])
        f = np.float32
        return dict(node=np.array([r.node for r in recs], np.int64),
                    stop=np.array([list(r.impact.stop) for r in recs], f),
                    stop_time=np.array([r.impact.stop_time for r in recs], f),
                    probability=np.array([r.probability for r in recs], f),
                    field_before=np.array([list(r.field_before) for r in recs], f),
                    phi_after=np.array([r.phi_after for r in recs], f),
                    field_after=np.array([list(r.field_after) for r in recs], f),
                    normal=np.array([list(r.normal) for r in recs], f))
    loss = s["learner"].train(case["steps"], batch=case["batch"], lr=1e-3, seed=s["seed"])
    return dict(loss=np.float32(loss), params=s["learner"].params())


# ---- what a pass cannot do without ------------------------------------------

def work(case):
    """Bytes and operations: each input of the mesh read once and each output
    written once.  A relaxation reads its system (column and coupling, the
    row's potential and right-hand side) for the correction and for the test
    that ends it; a sweep reads it once; fields read neighbours' positions
    and potentials once per row; a flight reads the tetrahedra on its way
    (about 178 accepted steps of an ion)."""
    mesh, a = _mesh(case)
    n, nnz = mesh.num_nodes, mesh.nnz
    dirichlet = np.isin(a["type"], [t for t, v in a["types"].items() if v["dirichlet"]])
    free = ~dirichlet
    rows = int(free.sum())
    entries = int(np.diff(a["row_ptr"])[free].sum())
    system = 12.0 * entries + 36.0 * rows
    fields = 24.0 * rows + 5.0 * entries + 24.0 * n
    flight, flight_ops = 178 * 224.0, 178 * 6 * 150.0
    kind = case["kind"]
    if kind == "event":
        per = (2 * system if case["relax_mode"] == 1 else system) + fields + flight
        return dict(bytes=case["count"] * per, flops=case["count"] * (4.0 * entries + flight_ops))
    if kind == "trace":
        return dict(bytes=fields + case["ions"] * flight, flops=case["ions"] * flight_ops + 30.0 * entries)
    if kind == "relax":
        return dict(bytes=2 * system + fields + 8.0 * n, flops=4.0 * entries)
    if kind == "sweep":
        return dict(bytes=case["cycles"] * system, flops=2.0 * case["cycles"] * entries)
    if kind == "snapshot":
        return dict(bytes=28.0 * n + 64.0 * n + 12.0 * nnz, flops=60.0 * nnz)
    if kind == "tips":
        return dict(bytes=case["tips"] * (2 * system + fields + flight),
                    flops=case["tips"] * (4.0 * entries + flight_ops))
    cells = 8 * case["batch"] * 580.0
    macs = 16 * 64 + 4 * 128 * 64
    return dict(bytes=case["steps"] * cells * (16 * 4 + 64 * 8), flops=6.0 * case["steps"] * cells * macs)


# ---- 64-bit values ------------------------------------------------------------

def _relaxed(a, types, phi):
    """The finite-volume solution in 64 bits: diagonally preconditioned
    conjugate gradients on the free cells, to the last digits.  A free cell
    that is not Neumann leaves its Neumann neighbours out of its sums."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    row = np.repeat(np.arange(len(types)), np.diff(a["row_ptr"]))
    col = a["col"].astype(np.int64)
    neumann = np.isin(types, [t for t, v in a["types"].items() if v["neumann"]])
    free = ~np.isin(types, [t for t, v in a["types"].items() if v["dirichlet"]])
    # every species of these specimens has permittivity 1, so a cell that
    # turns to vacuum keeps its couplings, save those with Neumann cells
    gone = types != a["type"]
    c = np.where((~neumann[row] & neumann[col]) | (neumann[row] & gone[col]), 0.0, a["coupling"])
    phi = phi.copy()

    def part(mask, rhs_phi):
        """Solves the rows of mask, every other cell held."""
        index = np.full(len(types), -1, np.int64)
        index[mask] = np.arange(mask.sum())
        m = int(mask.sum())
        use = mask[row]
        diag = np.bincount(index[row[use]], weights=c[use], minlength=m)
        inner = use & mask[col]
        held = use & ~mask[col]
        b = np.bincount(index[row[held]], weights=c[held] * rhs_phi[col[held]], minlength=m)
        crow = np.concatenate([[0], np.cumsum(np.bincount(index[row[inner]], minlength=m))])
        A = torch.sparse_csr_tensor(torch.tensor(crow), torch.tensor(index[col[inner]]), torch.tensor(c[inner]),
                                    size=(m, m), dtype=torch.float64).to(dev)
        d = torch.tensor(diag).to(dev)
        rhs = torch.tensor(b).to(dev)
        x = torch.zeros_like(d)
        r = rhs.clone()
        z = r / d
        p = z.clone()
        rz = torch.dot(r, z)
        stop = 1e-14 * float(torch.linalg.norm(rhs))
        for k in range(6000):
            ap = d * p - A @ p
            alpha = rz / torch.dot(p, ap)
            x += alpha * p
            r -= alpha * ap
            if k % 50 == 49 and float(torch.linalg.norm(r)) <= stop:
                break
            z = r / d
            new = torch.dot(r, z)
            p = z + (new / rz) * p
            rz = new
        return x.cpu().numpy()

    # the Neumann rows do not act on the others: one after the other
    v = free & ~neumann
    phi[v] = part(v, phi)
    w = free & neumann
    if w.any():
        phi[w] = part(w, phi)
    return phi


def _fields(a, types, phi, nodes=None):
    """field_o1 in 64 bits: the least-squares gradient over the neighbours
    with a coupling; zero on the hull."""
    n = len(phi)
    row = np.repeat(np.arange(n), np.diff(a["row_ptr"]))
    col = a["col"]
    neumann = np.isin(types, [t for t, v in a["types"].items() if v["neumann"]])
    gone = types != a["type"]
    use = (a["coupling"] != 0.0) & ~(neumann[row] & gone[col]) & ~(gone[row] & neumann[col])
    if nodes is not None:
        keep = np.zeros(n, bool)
        keep[nodes] = True
        use &= keep[row]
    row, col = row[use], col[use]
    x = a["xyz"].astype(np.float64)
    d = x[col] - x[row]
    dp = phi[col] - phi[row]
    M = np.zeros((n, 3, 3))
    b = np.zeros((n, 3))
    for i in range(3):
        b[:, i] = np.bincount(row, weights=dp * d[:, i], minlength=n)
        for j in range(3):
            M[:, i, j] = np.bincount(row, weights=d[:, i] * d[:, j], minlength=n)
    live = (a["hull"] == 0) if nodes is None else keep & (a["hull"] == 0)
    E = np.zeros((n, 3))
    scale = np.trace(M[live], axis1=1, axis2=2)
    E[live] = -np.linalg.solve(M[live] / scale[:, None, None], (b[live] / scale[:, None])[:, :, None])[:, :, 0]
    return E


def _surface(a, types):
    row = np.repeat(np.arange(len(types)), np.diff(a["row_ptr"]))
    removable = np.isin(types, [t for t, v in a["types"].items() if v["removable"]])
    return np.unique(row[removable[row] & (types[a["col"]] == VACUUM) & (a["area_pos"] > 0)])


def _probability(a, types, E, cells):
    ef = np.array([float(np.float32(a["types"][int(t)]["evap_field"])) for t in types[cells]])
    ratio = np.linalg.norm(E[cells], axis=1) / ef
    return ratio / ratio.sum()


def exact(case, seed):
    """Flights, plane-fit normals, training and runs of several events have no
    such value; relaxations, fields and the state of a single event do."""
    kind = case["kind"]
    single = kind == "event" and case["count"] == 1 and case["relax_mode"] == 1
    if kind not in ("relax", "snapshot") and not single:
        return None
    _, a = _mesh(case)
    types = a["type"].copy()
    types[_gone(a, seed)] = VACUUM
    start = _start(a, seed) if kind == "relax" else a["phi"].astype(np.float64)
    phi = _relaxed(a, types, start)
    if kind == "relax":
        return dict(phi=phi, field=_fields(a, types, phi))
    cells = _surface(a, types)
    if kind == "snapshot":
        E = _fields(a, types, phi)
        p = np.zeros(len(types))
        p[cells] = _probability(a, types, E, cells)
        return dict(phi=phi, field=E, force=None, types=None, probability=p, normal=None)
    E = _fields(a, types, phi, cells)
    p = _probability(a, types, E, cells)
    node = int(cells[np.argmax(p)])
    types[node] = VACUUM
    after = _relaxed(a, types, phi)
    return dict(node=None, id=None, voltage=None, stop=None, tof=None, probability=np.array([p.max()]),
                potential_before=phi[[node]], field_before=E[[node]], potential_after=after[[node]],
                field_after=_fields(a, types, after, [node])[[node]], normal=None, apex=None)
