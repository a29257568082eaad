"""Measured cases of the assemble-and-solve path, through the package's public calls.

Each case builds a model the way a user does (nodes, beams, holds, loads,
constraints, cost elements), keeps one `DeviceModel` for it, and passes host
arrays through one public call:

* assemble  one assembly of Lλ and Lλx.nzval (`DeviceModel.assemble`),
* sweep     a whole SweepX{0} or SweepX{2} solve (`DeviceModel.sweepx`),
* adjoint   cost and gradient of an identification (`DeviceModel.adjoint`),
* results   element results of every beam (`DeviceModel.beam_results`).

Models: "cantilever", a clamped beam; "lattice", a 3D frame held at its base;
"risers", vertical risers moved at the top; "batch", independent cantilevers and
portal frames; "identification", a simply supported beam with an EI scale per
element.  `exact` restates the element and the solves in 64 bits, with
derivatives by automatic differentiation.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "muscade.jl_gb300"))

FIELDS = ("t1", "t2", "t3", "r1", "r2", "r3")


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest call: one Newton iteration's assembly of a 20-beam cantilever
        dict(name="assemble cantilever 20", do="assemble", model="cantilever", nel=20, length=10.0, mission="static"),
        # a ragged frame in a Newmark step's first iteration, with hydrodynamic loads
        dict(name="assemble frame 13x11x7 step", do="assemble", model="lattice", nx=13, ny=11, nz=7, mission="step", drag=True),
        # riser analysis: a Newmark iteration of 200 risers of 250 beams, mass only
        dict(name="assemble risers 200x250 iter", do="assemble", model="risers", nriser=200, nel=250, mission="iter", drag=False),
        # the large frame: 210,000 beams, static
        dict(name="assemble lattice 60x60x20", do="assemble", model="lattice", nx=60, ny=60, nz=20, mission="static", drag=False),
        # a small static analysis from start to end, ten load steps
        dict(name="sweep cantilever 20", do="sweep", model="cantilever", nel=20, length=10.0, nstep=10),
        # a small space frame's first load step
        dict(name="sweep frame 6x5x4", do="sweep", model="lattice", nx=6, ny=5, nz=4, nstep=1, drag=False),
        # a middling space frame's static analysis
        dict(name="sweep frame 12x12x6", do="sweep", model="lattice", nx=12, ny=12, nz=6, nstep=3, drag=False),
        # the large frame's first load step
        dict(name="sweep lattice 60x60x20", do="sweep", model="lattice", nx=60, ny=60, nz=20, nstep=1, drag=False),
        # time stepping of 200 risers, three Newton iterations a step
        dict(name="sweep risers 200x250", do="sweep", model="risers", nriser=200, nel=250, nstep=4, drag=False),
        # a design study: uneven independent models, each with its own convergence
        dict(name="sweep batch 512", do="sweep", model="batch", nmodel=512, nmin=10, nmax=400, nstep=4),
        # stiffness identification: the gradient by the adjoint over a stretch of the record
        dict(name="adjoint 5000x12", do="adjoint", model="identification", nel=5000, nstep=12),
        # element results of some stored states
        dict(name="results risers 200x250", do="results", model="risers", nriser=200, nel=250, nstate=2, drag=False),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    do = rng.choice(["assemble", "assemble", "sweep", "sweep", "adjoint", "results"])
    if do == "adjoint":
        return dict(do=do, model="identification", nel=log(60, 4000), nstep=rng.randint(4, 12))
    if do == "results":
        return dict(do=do, model="risers", nriser=log(1, 200), nel=rng.randint(9, 250), nstate=rng.randint(1, 2), drag=rng.random() < 0.5)
    model = rng.choice(["cantilever", "lattice", "risers", "batch"] if do == "sweep" else ["cantilever", "lattice", "risers"])
    if model == "cantilever":
        c = dict(do=do, model=model, nel=log(5, 400), length=2.0)
    elif model == "lattice":
        top = 60 if do == "assemble" else 36
        c = dict(do=do, model=model, nx=log(3, top), ny=log(3, top), nz=log(3, 20 if do == "assemble" else 12), drag=False)
    elif model == "risers":
        c = dict(do=do, model=model, nriser=log(1, 200), nel=rng.randint(40, 250), drag=rng.random() < 0.5)
    else:
        c = dict(do=do, model=model, nmodel=log(4, 400), nmin=10, nmax=rng.randint(100, 400))
    if do == "assemble":
        c["mission"] = rng.choice(["static", "step", "iter"])
        if model == "lattice":
            c["drag"] = rng.random() < 0.5
    else:
        c["nstep"] = 1 if model == "lattice" else rng.randint(1, 4)
    return c


# ------------------------------------------------------------------ geometry and values of a model
def _rng(case, seed):
    return np.random.Generator(np.random.PCG64([int(seed) & 0x7FFFFFFF, 2026]))


def _section(rng, n, EA, EI, GJ, mu, iota1, sigma, drag=False):
    ln = np.exp(rng.normal(0.0, sigma, (4, n)))
    s = dict(EA=EA * ln[0], EI2=EI * ln[1], EI3=EI * ln[2], GJ=GJ * ln[3], mu=np.full(n, mu), iota1=np.full(n, iota1))
    for k in ("w", "Ca1", "Cl1", "Cq1", "Ca2", "Cl2", "Cq2", "Ca3", "Cl3", "Cq3"):
        s[k] = np.zeros(n)
    if drag:  # submerged weight, added mass, linear and quadratic drag across the element
        s["w"][:] = 0.3 * mu
        for k, v in (("Ca2", mu), ("Ca3", mu), ("Cl1", 0.02 * mu), ("Cl2", 0.05 * mu), ("Cl3", 0.05 * mu), ("Cq2", 0.4 * mu), ("Cq3", 0.4 * mu)):
            s[k][:] = v
    return s


def _mesh(case, seed):
    """Everything that defines the model, as arrays: nodes xyz, beams (0-based node
    pairs, orient2, section), holds [(field, nodes)], loads [(field, nodes, amplitude)]
    ramped by t, prescribed [(field, nodes, amplitude, period)], lines (node chains)."""
    rng = _rng(case, seed)
    m = dict(holds=[], loads=[], prescribed=[], dynamic=False)
    kind = case["model"]
    if kind == "cantilever":
        nel = case["nel"]
        m["xyz"] = np.stack([np.linspace(0.0, case["length"], nel + 1), np.zeros(nel + 1), np.zeros(nel + 1)], axis=1)
        m["conn"] = np.stack([np.arange(nel), np.arange(1, nel + 1)], axis=1)
        m["orient"] = np.tile([0.0, 1.0, 0.0], (nel, 1))
        m["section"] = {k: np.full(nel, v[0]) for k, v in _section(rng, 1, 1e8, 1e4, 1e4, 10.0, 1.0, 0.05).items()}
        m["holds"] = [(f, np.array([0])) for f in FIELDS]
        m["loads"] = [("t3", np.array([nel]), np.array([1e3 * rng.uniform(0.95, 1.05)]))]
        m["lines"] = [np.arange(nel + 1)]
    elif kind == "lattice":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        nid = np.arange(nx * ny * nz).reshape(nx, ny, nz, order="F")
        I, J, K = np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz), indexing="ij")
        m["xyz"] = np.stack([I.ravel(order="F"), J.ravel(order="F"), K.ravel(order="F")], axis=1).astype(np.float64)
        pairs = ((nid[:-1], nid[1:]), (nid[:, :-1], nid[:, 1:]), (nid[:, :, :-1], nid[:, :, 1:]))
        edges = [np.stack([a.ravel(order="F"), b.ravel(order="F")], axis=1) for a, b in pairs]
        m["conn"] = np.concatenate(edges)
        # orient2 by edge direction, so that no element starts a half turn away from the axes
        m["orient"] = np.concatenate([np.tile(o, (len(e), 1)) for o, e in zip(([0.0, 1.0, 0.0], [0.0, 0.0, 1.0], [1.0, 0.0, 0.0]), edges)])
        m["section"] = _section(rng, len(m["conn"]), 1e8, 1e4, 1e4, 10.0, 1.0, 0.1, case.get("drag", False))
        m["holds"] = [(f, nid[:, :, 0].ravel(order="F")) for f in FIELDS]
        free = nid[:, :, 1:].ravel(order="F")
        m["loads"] = [(f, free, rng.normal(0.0, 100.0, len(free))) for f in FIELDS[:3]]
    elif kind == "risers":
        nr, nel = case["nriser"], case["nel"]
        z = np.linspace(0.0, 4.0 * nel, nel + 1)
        r = np.repeat(np.arange(nr), nel + 1)
        m["xyz"] = np.stack([50.0 * (r % 20), 50.0 * (r // 20), np.tile(z, nr)], axis=1).astype(np.float64)
        first = np.arange(nr) * (nel + 1)
        m["conn"] = (first[:, None, None] + np.stack([np.arange(nel), np.arange(1, nel + 1)], axis=1)[None]).reshape(-1, 2)
        m["orient"] = np.tile([1.0, 0.0, 0.0], (len(m["conn"]), 1))
        m["section"] = _section(rng, len(m["conn"]), 5e9, 1e6, 1e6, 300.0, 10.0, 0.0, case["drag"])
        m["holds"] = [(f, first) for f in ("t1", "t2", "t3", "r1")]
        m["prescribed"] = [("t1", first + nel, rng.uniform(1.0, 5.0, nr), rng.uniform(8.0, 15.0, nr)),
                           ("t2", first + nel, np.zeros(nr), np.full(nr, 1.0)),
                           ("t3", first + nel, np.full(nr, 0.1), np.full(nr, math.inf))]
        m["lines"] = [f + np.arange(nel + 1) for f in first]
        m["dynamic"] = True
    elif kind == "batch":
        xyz, conn, held, loaded, amp, sec, lines, off = [], [], [], [], [], [], [], 0
        sizes = np.random.Generator(np.random.PCG64(2030))  # the study's models; sections and loads vary with the seed
        for i in range(case["nmodel"]):
            n = int(sizes.integers(case["nmin"], case["nmax"] + 1))
            x, hold, load, sign = _frame_model(sizes.random() < 0.5, n)
            x[:, 1] += 30.0 * i
            xyz.append(x)
            lines.append(off + np.arange(len(x)))
            conn.append(np.stack([lines[-1][:-1], lines[-1][1:]], axis=1))
            held += [off + h for h in hold]
            loaded.append(off + load)
            amp.append(sign * rng.gumbel(1e3, 200.0))
            sec.append({k: np.full(len(x) - 1, v[0]) for k, v in _section(rng, 1, 1e8, 1e4, 1e4, 10.0, 1.0, 0.15).items()})
            off += len(x)
        m["xyz"], m["conn"], m["lines"] = np.concatenate(xyz), np.concatenate(conn), lines
        m["orient"] = np.tile([0.0, 1.0, 0.0], (len(m["conn"]), 1))
        m["section"] = {k: np.concatenate([s[k] for s in sec]) for k in sec[0]}
        m["holds"] = [(f, np.array(held)) for f in FIELDS]
        m["loads"] = [("t3", np.array(loaded), np.array(amp))]
    else:  # identification
        nel, nstep = case["nel"], case["nstep"]
        x = 0.1 * np.arange(nel + 1)
        m["xyz"] = np.stack([x, np.zeros(nel + 1), np.zeros(nel + 1)], axis=1)
        m["conn"] = np.stack([np.arange(nel), np.arange(1, nel + 1)], axis=1)
        m["orient"] = np.tile([0.0, 1.0, 0.0], (nel, 1))
        m["section"] = _section(rng, nel, 1e10, 1e8, 1e8, 1e3, 10.0, 0.0)
        m["holds"] = [(f, np.array([0, nel])) for f in FIELDS[:3]] + [("r1", np.array([0]))]
        times = 0.01 * np.arange(1, nstep + 1)
        wx, wt, ph = rng.normal(0.0, 0.1, 16), rng.normal(0.0, 5.0, 16), rng.uniform(0.0, 2 * math.pi, 16)
        m["table"] = 1e3 * math.sqrt(2 / 16) * np.cos(wx * x[1:-1, None] + wt * times[:, None, None] + ph).sum(axis=2)
        m["sensors"] = np.sort(rng.choice(np.arange(1, nel), max(1, nel // 20), replace=False))
        m["record"] = rng.normal(0.0, 1e-4, (nstep, len(m["sensors"])))
        m["A"] = np.exp(rng.normal(0.0, 0.2, nel))
        m["lines"] = [np.arange(nel + 1)]
        m["dynamic"] = True
    return m


def _frame_model(portal, nel):
    """Nodes in line order, held nodes, loaded node and load sign of a 2 m cantilever
    or a portal frame (5 m columns, 10 m beam) of nel beams."""
    if not portal:
        return np.stack([np.linspace(0.0, 2.0, nel + 1), np.zeros(nel + 1), np.zeros(nel + 1)], axis=1), [0], nel, 1.0
    ncol = max(1, nel // 4)
    nb = nel - 2 * ncol
    if nb % 2:
        ncol, nb = ncol + 1, nb - 1
    s = np.concatenate([np.linspace(0.0, 5.0, ncol + 1), 5.0 + np.linspace(0.0, 10.0, nb + 1)[1:nb], 15.0 + np.linspace(0.0, 5.0, ncol + 1)])
    x = np.stack([np.clip(s - 5.0, 0.0, 10.0), np.zeros_like(s), np.minimum(np.minimum(s, 5.0), 20.0 - s)], axis=1)
    return x, [0, len(x) - 1], ncol + nb // 2, -1.0


def _ramp(t):
    return 0.5 * (1.0 - math.cos(math.pi * min(t, 5.0) / 5.0))


def _motion(t, amplitude, period):
    return amplitude * (np.sin(2 * math.pi * t / period) if np.all(np.isfinite(period)) else 1.0) * _ramp(t)


def _times(case):
    n = case["nstep"]
    return {"cantilever": 0.1, "lattice": 0.2, "risers": 0.05, "batch": 0.125, "identification": 0.01}[case["model"]] * np.arange(1, n + 1)


def _newmark(dt):
    return dict(a1=2 / dt, a2=2.0, a3=0.0, b1=4 / dt**2, b2=4 / dt, b3=2.0)  # β = 1/4, γ = 1/2


def _state_values(case, m, n, seed):
    """Random dof values of a state, for the calls that take one: displacements and
    rotations of a deformed structure, their rates, and multipliers."""
    rng = np.random.Generator(np.random.PCG64([int(seed) & 0x7FFFFFFF, 7]))
    k = case.get("nstate", 1 if case.get("mission") == "static" else 3)
    return rng.normal(0.0, 0.05, (k, n))


# ------------------------------------------------------------------ the package's side
def _model(case, m):
    from muscade_gpu.elements import BeamCrossSection, DofConstraint, DofLoad, EulerBeam3D, Hold, QuadraticCost, SingleAcost, SingleDofCost
    from muscade_gpu.model import Model

    model = Model(case["model"])
    nodes = model.addnode(m["xyz"])
    adof = case["model"] == "identification"
    conn = nodes[m["conn"]]
    if adof:
        pnodes = model.addnode(m["xyz"][:-1] + [0.05, 1.0, 0.0])
        conn = np.concatenate([conn, pnodes[:, None]], axis=1)
    cut = np.flatnonzero(np.any(np.diff(m["orient"], axis=0) != 0, axis=1)) + 1
    for a, b in zip([0, *cut], [*cut, len(conn)]):
        mat = BeamCrossSection(**{k: v[a:b] for k, v in m["section"].items()})
        model.addelement(EulerBeam3D, conn[a:b], mat=mat, orient2=tuple(m["orient"][a]), adof=adof)
    for f, at in m["holds"]:
        model.addelement(Hold, nodes[at][:, None], field=f)
    for i, (f, at, amplitude, period) in enumerate(m["prescribed"]):
        model.addelement(DofConstraint, nodes[at][:, None], xinod=(1,), xfield=(f,), lfield=f"λtop{i + 1}", coeffs=[1.0],
                         offset=lambda t, a=amplitude, p=period: _motion(t, a, p), name=f"top{i + 1}")
    for f, at, amplitude in m["loads"]:
        model.addelement(DofLoad, nodes[at][:, None], field=f, value=lambda t, a=amplitude: a * t)
    if adof:
        table, record = m["table"], m["record"]
        model.addelement(DofLoad, nodes[1:-1][:, None], field="t2", value=lambda t: table[int(round(t / 0.01)) - 1])
        for s, at in enumerate(m["sensors"]):
            y = record[:, s]
            model.addelement(SingleDofCost, [int(nodes[at])], cls="X", field="t2", cost=QuadraticCost(1e8, lambda t, y=y: y[int(round(t / 0.01)) - 1]))
        model.addelement(SingleAcost, pnodes[:, None], field="EIscale", cost=QuadraticCost(1.0, 1.0))
    return model


def prepare(case, seed):
    from muscade_gpu.device import DeviceModel

    m = _mesh(case, seed)
    model = _model(case, m)
    st = model.initialize(time=0.0)
    dm = DeviceModel(model, st.dis)
    s = dict(case=case, dm=dm)
    n = model.ndof["X"]
    if case["do"] == "assemble":
        s["X"] = list(_state_values(case, m, n, seed))
    elif case["do"] == "results":
        s["X"] = _state_values(case, m, n, seed)
    elif case["do"] == "sweep":
        s["X0"] = [np.zeros(n)] * (3 if m["dynamic"] else 1)
        s["times"] = _times(case)
    else:
        s["X0"] = [np.zeros(n)] * 3
        s["times"] = _times(case)
        s["tvals"] = dm.time_values(s["times"])  # loads and sensor records, tabulated once
        dm.set_A(m["A"])
    return s


def run(s):
    case, dm = s["case"], s["dm"]
    if case["do"] == "assemble":
        mission = ("static", "step", "iter").index(case["mission"])
        Ll, nz = dm.assemble(s["X"], t=0.5, mission=mission, c=_newmark(0.05) if mission else None, reuse=True)
        return {"Ll": Ll, "nzval": nz}
    if case["do"] == "results":
        return dm.beam_results(0, s["X"])
    if case["do"] == "adjoint":
        cost, dCdA, _, _ = dm.adjoint(2, s["times"], 0.0, s["X0"], maxdx=1e-7, tvals=s["tvals"])
        return {"cost": cost, "dCdA": dCdA}
    if case["model"] == "risers":
        rc, states, _ = dm.sweepx(2, s["times"], 0.0, s["X0"], fixed_iter=3)
    elif case["model"] == "batch":
        rc, states, _ = dm.sweepx(0, s["times"], 0.0, s["X0"], maxdx=1e-9, per_component=True)
    elif case["model"] == "cantilever":
        rc, states, _ = dm.sweepx(0, s["times"], 0.0, s["X0"], maxdx=1e-9)
    else:
        rc, states, _ = dm.sweepx(0, s["times"], 0.0, s["X0"], maxdx=1e-6, maxLl=1e-3)
    if rc:
        raise RuntimeError(dm.lib.mgpu_last_error(dm.ctx).decode())
    return states


# ------------------------------------------------------------------ work
def _counts(case):
    """Beams, X-dofs and stored entries of Lλx (about)."""
    kind = case["model"]
    if kind == "lattice":
        x, y, z = case["nx"], case["ny"], case["nz"]
        ne, nn = (x - 1) * y * z + x * (y - 1) * z + x * y * (z - 1), x * y * z
        nd = 6 * nn + 6 * x * y
    else:
        lines, nel = {"cantilever": (1, case.get("nel")), "identification": (1, case.get("nel")), "risers": (case.get("nriser"), case.get("nel")),
                      "batch": (case.get("nmodel"), 0.5 * (case.get("nmin", 0) + case.get("nmax", 0)))}[kind]
        ne, nn = lines * nel, lines * (nel + 1)
        nd = 6 * nn + 8 * lines
    return ne, nd, 72 * ne + 36 * nn


def work(case):
    """One pass's inputs and outputs in bytes; operations of the beams' residuals and
    tangents (2,000 a static beam, 6,000 with the time derivatives, at the least), of
    band factorisations (2 n b² with b = 12), and of nested dissection on the frames."""
    ne, nd, nnz = _counts(case)
    beam_bytes, solve = 50 * 8 + 13 * 4, 2 * nd * 12 * 12
    if case["do"] == "results":
        return {"bytes": case["nstate"] * (8 * nd + ne * 400) + ne * 69 * 8, "flops": case["nstate"] * ne * 1000}
    if case["do"] == "assemble":
        dyn = case["mission"] != "static"
        return {"bytes": ne * beam_bytes + 8 * nd * (4 if dyn else 2) + 8 * nnz, "flops": ne * (6000 if dyn else 2000)}
    dyn = case["model"] in ("risers", "identification")
    if case["model"] == "lattice":
        a, b, c = sorted((case["nx"], case["ny"], case["nz"]))
        solve = 8 * (6 * a * b) ** 3 * c / b + 2 * nd * 36
    per_step = {"risers": 3, "identification": 4}.get(case["model"], 3)
    its = case["nstep"] * per_step
    return {"bytes": its * (ne * beam_bytes + 8 * nnz) + 8 * nd * case["nstep"], "flops": its * (ne * (6000 if dyn else 2000) + solve)}


# ------------------------------------------------------------------ 64-bit restatement
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(x):
    return torch.as_tensor(np.asarray(x), dtype=torch.float64, device=_dev())


def _cross(a, b):
    return torch.cross(a, b.expand_as(a), dim=0)


def _rod(v):
    """Rotation matrix [i, column, n] of the rotation vectors v [3, n], by power series of |v|²."""
    s = v.square().sum(0)
    A = B = 0.0
    for k in range(12, -1, -1):
        A = 1.0 / math.factorial(2 * k + 1) - s * A
        B = 1.0 / math.factorial(2 * k + 2) - s * B
    S = torch.einsum("ikj,jn->ikn", _LEVI.to(v), v)
    eye = torch.eye(3, dtype=v.dtype, device=v.device)[:, :, None]
    return eye + A * S + B * (v[:, None] * v[None] - s * eye)


_LEVI = torch.zeros(3, 3, 3, dtype=torch.float64)  # spin(v)[i, k] = LEVI[i, k, j] v_j
for _i, _j, _k in ((0, 1, 2), (1, 2, 0), (2, 0, 1)):
    _LEVI[_i, _k, _j], _LEVI[_i, _j, _k] = 1.0, -1.0


def _log(M):
    """Rotation vector [3, n] of the rotations M [i, column, n]."""
    c = 0.5 * (M[0, 0] + M[1, 1] + M[2, 2] - 1.0)
    y = 1.0 - c
    near = y < 0.25
    yn, cf = torch.where(near, y, 0.1), torch.where(near, 0.0, c)
    f = 0.0
    for k in range(22, -1, -1):  # φ/sin φ = Σ (2y)ᵏ (k!)²/(2k+1)!
        f = 1.0 + f * yn * ((k + 1) / (2 * k + 3))
    f = torch.where(near, f, torch.acos(cf) / torch.sqrt(1.0 - cf * cf))
    return 0.5 * f * torch.stack([M[2, 1] - M[1, 2], M[0, 2] - M[2, 0], M[1, 0] - M[0, 1]])


def _mul(M, N):
    return (M[:, :, None] * N[None]).sum(1)  # [i, k, n] · [k, j, n]


def _vec(M, v):
    return (M * v[None]).sum(1)


def _tvec(M, v):
    return (M * v[:, None]).sum(0)


class _Beams:
    """Corotated beams, one per entry of the last axis: 4 Gauss points, strain energy
    and loads as functions of the element's dofs."""

    def __init__(self, m):
        c1, c2 = _t(m["xyz"][m["conn"][:, 0]]).T, _t(m["xyz"][m["conn"][:, 1]]).T
        o = _t(m["orient"]).T
        self.tg, self.cm = c2 - c1, 0.5 * (c1 + c2)
        L = self.L = self.tg.square().sum(0).sqrt()
        t = self.tg / L
        nv = o - t * (o * t).sum(0)
        nv = nv / nv.square().sum(0).sqrt()
        self.rm = torch.stack([t, nv, _cross(t, nv)], 1)
        s = self.s = {k: _t(v) for k, v in m["section"].items()}
        self.C = {k: torch.stack([s[f"{k}{i}"] for i in (1, 2, 3)])[None] for k in ("Ca", "Cl", "Cq")}
        r65, r30 = math.sqrt(6 / 5), math.sqrt(30.0)
        z = _t([-0.5 * math.sqrt(3 / 7 + 2 / 7 * r65), -0.5 * math.sqrt(3 / 7 - 2 / 7 * r65)])
        z = self.z = torch.cat([z, -z.flip(0)])[:, None]
        w = [(18 - r30) / 72, (18 + r30) / 72]
        self.w = _t(w + w[::-1])[:, None] * L  # [point, n]
        self.ya, self.yu, self.yv = 2 * z + 0 * L, 3 * z - 4 * z**3 + 0 * L, (z * z - 0.25) * L
        self.ka, self.ku = 2.0 / L, -24 * z / L**2

    def frame(self, X):
        r1, r2 = _rod(X[3:6]), _rod(X[9:12])
        dv = 0.5 * _log(_mul(r2, r1.transpose(0, 1)))
        rs = _mul(_rod(dv), _mul(r1, self.rm))
        d = 0.5 * (X[6:9] - X[0:3]) + 0.5 * self.tg
        return rs, dv, d

    def points(self, X, rs, dv, d):
        """Positions [point, 3, n]."""
        th, w = _tvec(rs, dv), _tvec(rs, d)
        p = torch.stack([self.L * self.z + self.ya * (w[0] - 0.5 * self.L), self.yu * w[1] + self.yv * th[2], self.yu * w[2] - self.yv * th[1]])
        return (rs[:, :, None] * p[None]).sum(1).transpose(0, 1) + (0.5 * (X[0:3] + X[6:9]) + self.cm)[None]

    def strains(self, X, rs, dv, d):
        """ε [n] and curvatures [3, point, n]."""
        th, w = _tvec(rs, dv), _tvec(rs, d)
        eps = 2 * d.square().sum(0).sqrt() / self.L - 1.0
        ka = self.ka + 0 * self.z
        return eps, torch.stack([ka * th[0], self.ku * w[1] + ka * th[2], self.ku * w[2] - ka * th[1]])

    def residual(self, X0, X1=None, X2=None, A=1.0):
        """R [12, n]: the gradient of strain energy and load potential, loads held."""
        s = self.s
        dyn = X1 is not None
        if dyn:
            def at(X):
                rs, dv, d = self.frame(X)
                return torch.cat([self.points(X, rs, dv, d), rs.transpose(0, 1)])  # points, then t, n, b

            def rate(X, V):
                return torch.func.jvp(at, (X,), (V,))[1]

            q2, q1 = (lambda r: (r[1], r[0]))(torch.func.jvp(rate, (X0, X1), (X1, X2)))
            rs = self.frame(X0)[0]
            v, a = q1[:4], q2[:4]
            vl, al = [(q[:, :, None] * rs[None]).sum(1) for q in (v, a)]  # [point, axis, n]
            fl = self.C["Ca"] * al + self.C["Cl"] * vl + self.C["Cq"] * vl * vl.abs()
            loads = s["mu"] * a + (rs[None] * fl[:, None]).sum(2) + s["w"] * _t([0.0, 0.0, 1.0])[None, :, None]
            spin = 0.5 * ((rs[:, 2] * q2[5]).sum(0) - (rs[:, 1] * q2[6]).sum(0))
            me = s["iota1"] * spin * rs[:, 0]

        def potential(X):
            rs, dv, d = self.frame(X)
            eps, kap = self.strains(X, rs, dv, d)
            xg = self.points(X, rs, dv, d)
            e = 0.5 * (s["EA"] * eps**2 + s["GJ"] * kap[0] ** 2 + A * (s["EI3"] * kap[1] ** 2 + s["EI2"] * kap[2] ** 2))
            P = (self.w * (e + ((loads * xg).sum(1) if dyn else s["w"] * xg[:, 2]))).sum()
            return P + (self.L * (me * _log(rs)).sum(0)).sum() if dyn else P

        return torch.func.grad(potential)(X0)

    def tangent(self, X, p, A=1.0):
        """∂R/∂(dof j) along (p0, p1, p2) of (X, X′, X″): [12 (i), 12 (j), n]."""
        def column(e):
            e = e[:, None].expand_as(X[0])
            return torch.func.jvp(lambda *x: self.residual(*x, A=A), tuple(X), tuple(q * e for q in p))[1]

        return torch.func.vmap(column, out_dims=1)(torch.eye(12, dtype=torch.float64, device=_dev()))

    def results(self, X):
        rs, dv, d = self.frame(X)
        eps, kap = self.strains(X, rs, dv, d)
        x, s = self.points(X, rs, dv, d), self.s
        k = kap.permute(2, 1, 0)
        mi = k * torch.stack([s["GJ"], s["EI3"], s["EI2"]], -1)[:, None]
        return dict(eps=eps, rsm=rs.permute(2, 0, 1), x=x.permute(2, 0, 1), kappa=k, fi=(s["EA"] * eps)[:, None].expand(-1, 4), mi=mi)


def _numbering(m):
    """X-dofs (0-based) of the beams and of the multipliers: nodes in the order the
    beams name them, six dofs each, then one multiplier per hold and constraint."""
    flat = m["conn"].ravel()
    _, first = np.unique(flat, return_index=True)
    rank = np.zeros(len(m["xyz"]), dtype=np.int64)
    rank[flat[np.sort(first)]] = np.arange(len(first))
    n = 6 * len(first)
    cons = []  # (dof, multiplier, amplitude, period) per hold or constraint group
    for f, at, amplitude, period in [(f, at, None, None) for f, at in m["holds"]] + m["prescribed"]:
        cons.append((6 * rank[at] + FIELDS.index(f), n + np.arange(len(at)), amplitude, period))
        n += len(at)
    edof = np.concatenate([6 * rank[m["conn"][:, [0]]] + np.arange(6), 6 * rank[m["conn"][:, [1]]] + np.arange(6)], axis=1)
    loads = [(6 * rank[at] + FIELDS.index(f), amplitude) for f, at, amplitude in m["loads"]]
    return rank, edof, cons, loads, n


def _offset(t, amplitude, period, n):
    return np.zeros(n) if amplitude is None else _motion(t, amplitude, period)


def _exact_assemble(case, seed):
    m = _mesh(case, seed)
    rank, edof, cons, loads, n = _numbering(m)
    X = _t(_state_values(case, m, n, seed))
    d = torch.as_tensor(edof, device=_dev())
    beams, t = _Beams(m), 0.5
    Xe = [x[d.T] for x in X]
    c = _newmark(0.05)
    p = (1.0,) if case["mission"] == "static" else (1.0, c["a1"], c["b1"])
    Re, Ke = beams.residual(*Xe), beams.tangent(Xe, p)
    if case["mission"] == "step":
        a, b = [c[k + "2"] * Xe[1] + c[k + "3"] * Xe[2] for k in "ab"]
        Re = Re - torch.func.jvp(beams.residual, tuple(Xe), (torch.zeros_like(a), a, b))[1]
    Ll = torch.zeros(n, dtype=torch.float64, device=_dev())
    Ll.index_add_(0, d.T.reshape(-1), Re.reshape(-1))
    keys = [(d[:, None, :] * n + d[:, :, None]).reshape(-1)]  # column·n + row, [element, i, j]
    vals = [Ke.permute(2, 0, 1).reshape(-1)]
    x = X[0]
    for dof, lam, amplitude, period in cons:
        i, l = torch.as_tensor(dof, device=_dev()), torch.as_tensor(lam, device=_dev())
        Ll.index_add_(0, i, -x[l])
        Ll.index_add_(0, l, -(x[i] - _t(_offset(t, amplitude, period, len(dof)))))
        one = torch.ones(len(dof), dtype=torch.float64, device=_dev())
        for r, q, v in ((i, i, 0.0), (i, l, -1.0), (l, i, -1.0), (l, l, 0.0)):
            keys.append(q * n + r)
            vals.append(v * one)
    for dof, amplitude in loads:
        i = torch.as_tensor(dof, device=_dev())
        Ll.index_add_(0, i, -_t(amplitude) * t)
        keys.append(i * n + i)
        vals.append(torch.zeros(len(dof), dtype=torch.float64, device=_dev()))
    u, inv = torch.unique(torch.cat(keys), return_inverse=True)
    nz = torch.zeros(len(u), dtype=torch.float64, device=_dev()).index_add_(0, inv, torch.cat(vals))
    return {"Ll": Ll.cpu().numpy(), "nzval": nz.cpu().numpy()}


class _Lines:
    """Chains of beams, padded to one length: block-tridiagonal solves of 6 × 6 blocks
    over the free dofs (held and prescribed dofs get an identity row)."""

    def __init__(self, m):
        self.m, self.beams = m, _Beams(m)
        self.rank, self.edof, self.cons, self.loads, self.n = _numbering(m)
        lines = m["lines"]
        self.nl, self.nn = len(lines), max(len(q) for q in lines)
        self.d = torch.as_tensor(self.edof, device=_dev())
        place = np.full(6 * len(m["xyz"]), -1)
        for r, q in enumerate(lines):
            for f in range(6):
                place[6 * self.rank[q] + f] = (r * self.nn + np.arange(len(q))) * 6 + f
        self.place = torch.as_tensor(place, device=_dev())  # dof -> padded position
        self.blk = self.place[self.d[:, 0]] // 6  # first node's padded block of every beam
        self.nd = len(place)
        self.held = torch.as_tensor(np.concatenate([c[0] for c in self.cons]), device=_dev())
        self.lam = torch.as_tensor(np.concatenate([c[1] for c in self.cons]), device=_dev())
        self.free = torch.ones(self.nl * self.nn * 6, dtype=torch.bool, device=_dev())
        self.free[self.place[self.held]] = False

    def offsets(self, t):
        return _t(np.concatenate([_offset(t, a, p, len(i)) for i, _, a, p in self.cons]))

    def factor(self, K):
        """Block LU of the assembled matrix of element matrices K [12, 12, ne]."""
        nb, k = self.nl * self.nn, K.permute(2, 0, 1)
        D = torch.zeros(nb, 6, 6, dtype=torch.float64, device=_dev())
        D.index_add_(0, self.blk, k[:, :6, :6].contiguous())
        D.index_add_(0, self.blk + 1, k[:, 6:, 6:].contiguous())
        U, Lo = torch.zeros_like(D), torch.zeros_like(D)
        U[self.blk], Lo[self.blk + 1] = k[:, :6, 6:], k[:, 6:, :6]
        f = self.free.reshape(nb, 6).to(torch.float64)
        fp = torch.cat([f[1:], f[:1]])
        fm = torch.cat([f[-1:], f[:-1]])
        D = D * f[:, :, None] * f[:, None, :]
        U, Lo = U * f[:, :, None] * fp[:, None, :], Lo * f[:, :, None] * fm[:, None, :]
        pad = torch.zeros(self.nl * self.nn * 6, dtype=torch.bool, device=_dev())
        pad[self.place] = True
        D = D + torch.diag_embed(1.0 - f * pad.reshape(nb, 6))
        D, U, Lo = [q.reshape(self.nl, self.nn, 6, 6).unbind(1) for q in (D, U, Lo)]
        G, inv = [], None
        for i in range(self.nn):
            Di = D[i] if i == 0 else D[i] - Lo[i] @ (inv @ U[i - 1])
            inv = torch.linalg.inv(Di)
            G.append(inv)
        return G, U, Lo

    def solve(self, fac, b, transposed=False):
        """x with A x = b (or Aᵀ x = b), b over the dofs; zero at held dofs."""
        G, U, Lo = fac
        if transposed:
            G = [g.mT for g in G]
            U, Lo = [q.mT for q in [*Lo[1:], Lo[0]]], [q.mT for q in [U[-1], *U[:-1]]]
        r = torch.zeros(self.nl * self.nn * 6, dtype=torch.float64, device=_dev())
        r[self.place] = b
        r = (r * self.free).reshape(self.nl, self.nn, 6, 1).unbind(1)
        y = [r[0]]
        for i in range(1, self.nn):
            y.append(r[i] - Lo[i] @ (G[i - 1] @ y[-1]))
        x = [None] * self.nn
        x[-1] = G[-1] @ y[-1]
        for i in range(self.nn - 2, -1, -1):
            x[i] = G[i] @ (y[i] - U[i] @ x[i + 1])
        return torch.stack(x, 1).reshape(-1)[self.place]

    def gather(self, R):
        return torch.zeros(self.nd, dtype=torch.float64, device=_dev()).index_add_(0, self.d.T.reshape(-1), R.reshape(-1))

    def apply(self, K, v):
        return self.gather((K * v[self.d.T][None]).sum(1))

    def step(self, x, rates, lam, f, t, dt, first, A=1.0):
        """One Newton iteration of SweepX: the new x, rates, multipliers and Δx."""
        c = _newmark(dt) if rates else None
        Xe = [q[self.d.T] for q in (x, *rates)]
        R, K = self.beams.residual(*Xe, A=A), self.beams.tangent(Xe, (1.0, c["a1"], c["b1"]) if rates else (1.0,), A=A)
        if rates and first:
            a, b = [c[k + "2"] * rates[0] + c[k + "3"] * rates[1] for k in "ab"]
            R = R - torch.func.jvp(lambda *q: self.beams.residual(*q, A=A), tuple(Xe), (torch.zeros_like(Xe[0]), a[self.d.T], b[self.d.T]))[1]
        r = self.gather(R) - f
        g = torch.zeros_like(x)
        g[self.held] = x[self.held] - self.offsets(t)  # Δx of the held dofs
        fac = self.factor(K)
        dx = g + self.solve(fac, r - self.apply(K, g))
        lam = (r - self.apply(K, dx))[self.held]
        if rates:
            da, db = c["a1"] * dx, c["b1"] * dx
            if first:
                da, db = da + a, db + b
            rates = [rates[0] - da, rates[1] - db]
        else:
            rates = []
        return x - dx, rates, lam, dx, fac


def _line_cost(case):
    """Seconds that a chain's sweeps take, about."""
    nn = {"batch": case.get("nmax", 0)}.get(case["model"], case.get("nel", 0))
    its = {"cantilever": 8, "risers": 3, "batch": 14}.get(case["model"], 3) * case["nstep"]
    once = nn * 4e-4 + (0.6 if case["model"] in ("risers", "identification") else 0.2)
    return its * once + (case["nstep"] * (nn * 3e-4 + 1.0) if case["do"] == "adjoint" else 0.0)


def _exact_sweep(case, seed):
    L = _Lines(_mesh(case, seed))
    x = torch.zeros(L.nd, dtype=torch.float64, device=_dev())
    rates = [torch.zeros_like(x), torch.zeros_like(x)] if L.m["dynamic"] else []
    lam = torch.zeros(len(L.held), dtype=torch.float64, device=_dev())
    out, told = [], 0.0
    for t in _times(case):
        f = torch.zeros_like(x)
        for dof, amplitude in L.loads:
            f.index_add_(0, torch.as_tensor(dof, device=_dev()), _t(amplitude) * t)
        for it in range(3 if L.m["dynamic"] else 50):
            x, rates, lam, dx, _ = L.step(x, rates, lam, f, t, t - told, it == 0)
            if not L.m["dynamic"] and float(dx.abs().max()) < 1e-9:
                break
        told = t
        rows = []
        for k, q in enumerate((x, *rates)):
            full = torch.zeros(L.n, dtype=torch.float64, device=_dev())
            full[: L.nd] = q
            if k == 0:
                full[L.lam] = lam
            rows.append(full)
        if rates:  # the rates of the multipliers follow the same update from zero
            c = _newmark(0.05)
            old = out[-1] if out else torch.zeros(3, L.n, dtype=torch.float64, device=_dev())
            dl = old[0][L.lam] - lam
            rows[1][L.lam] = old[1][L.lam] - (c["a1"] * dl + c["a2"] * old[1][L.lam] + c["a3"] * old[2][L.lam])
            rows[2][L.lam] = old[2][L.lam] - (c["b1"] * dl + c["b2"] * old[1][L.lam] + c["b3"] * old[2][L.lam])
        out.append(torch.stack(rows))
    return torch.stack(out).cpu().numpy()


def _exact_adjoint(case, seed):
    m = _mesh(case, seed)
    L = _Lines(m)
    A = _t(m["A"])
    times = _times(case)
    dt = times[0]
    c = _newmark(dt)
    inner = torch.as_tensor(6 * L.rank[1:-1] + 1, device=_dev())
    sens = torch.as_tensor(6 * L.rank[m["sensors"]] + 1, device=_dev())
    y, table = _t(m["record"]), _t(m["table"])
    zero = torch.zeros(L.nd, dtype=torch.float64, device=_dev())
    x, rates, lam, cost, kept = zero, [zero, zero], None, 0.0, []
    for k, t in enumerate(times):
        f = zero.clone()
        f[inner] = table[k]
        for it in range(12):
            x, rates, lam, dx, fac = L.step(x, rates, lam, f, t, dt, it == 0, A=A)
            if it and float(dx.abs().max()) < 1e-8:
                break
        r = x[sens] - y[k]
        cost = cost + dt * 1e8 * r.square().sum()
        kept.append((x, rates, fac, 2 * dt * 1e8 * r))
    cost = cost + (A - 1.0).square().sum()
    g = 2 * (A - 1.0)
    xb, vb, ab = zero, zero, zero
    for x, rates, fac, r in reversed(kept):
        xb = xb.clone()
        xb[sens] += r
        mu = L.solve(fac, xb + c["a1"] * vb + c["b1"] * ab, transposed=True)
        Xe, me = [q[L.d.T] for q in (x, *rates)], mu[L.d.T]
        g = g - (me * torch.func.jvp(lambda a: L.beams.residual(*Xe, A=a), (A,), (torch.ones_like(A),))[1]).sum(0)

        def back(k):  # (∂R/∂X⁽ᵏ⁾)ᵀ μ
            return L.gather(torch.func.vjp(lambda q: L.beams.residual(*[q if i == k else Xe[i] for i in range(3)], A=A), Xe[k])[1](me)[0])

        # x′ = a1 (x − x₋) − (a2 − 1) x′₋ − a3 x″₋ and x″ alike, with R(x, x′, x″) = 0
        cv, ca = vb - back(1), ab - back(2)
        xb, vb, ab = (-c["a1"] * cv - c["b1"] * ca, (1 - c["a2"]) * cv - c["b2"] * ca, -c["a3"] * cv + (1 - c["b3"]) * ca)
    return {"cost": float(cost), "dCdA": g.cpu().numpy()}


def exact(case, seed):
    if case["do"] == "assemble":
        return _exact_assemble(case, seed)
    if case["do"] == "results":
        m = _mesh(case, seed)
        _, edof, _, _, n = _numbering(m)
        X, d, beams = _t(_state_values(case, m, n, seed)), torch.as_tensor(edof.T, device=_dev()), _Beams(m)
        got = [beams.results(x[d]) for x in X]
        return {k: torch.stack([g[k] for g in got]).cpu().numpy() for k in got[0]}
    if case["model"] == "lattice" or _line_cost(case) > 20:
        return None  # a 3D frame's sparse solve, or long chains: too long here
    return _exact_adjoint(case, seed) if case["do"] == "adjoint" else _exact_sweep(case, seed)
