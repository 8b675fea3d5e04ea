"""Performance cases: the work a program gives this framework, through its
public entry points (heliocubed_b200.Shell, O4Batch, Ensemble, AmrStep).

    listed()            the named cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) inputs on the GPU and the handles a program keeps
    run(state)          one pass and its outputs
    work(case)          bytes and FP64 operations one pass cannot do without
    exact(case, seed)   the outputs from plain torch in 64 bits

Inputs are a Parker-like solar wind with seeded tangential perturbations of v
and B, a current sheet at the equator, a seeded pressure pulse and, with
`cloud`, a seeded spherical cloud (denser and faster, with jumps that reach
the limiters, the WENOZ detector and the Roe fan check).  A pass of the level
cases starts from the initial state again (one device copy), so that every
pass meets these fields and not the relaxed wind.
"""
import math
import random

import numpy as np
import torch

import heliocubed_b200 as hc
from heliocubed_b200.amr import AmrStep
from heliocubed_b200.level import Ensemble, O4Batch, make_box

GAMMA = 5.0 / 3.0
MP = 1.67262192e-24
RHO_FLOOR = MP / 100
RSUN = 6.96e10
GM = 6.67430e-8 * 1.98847e33
R_IN, R_OUT, STRETCH = 21.5 * RSUN, 215.0 * RSUN, 1.5
ENTROPY, ETA_D, CFL = 0.3, 0.02, 0.4
PI = math.pi
PERM = ((1, 2, 0), (1, 2, 0), (1, 0, 2), (0, 1, 2), (1, 0, 2), (0, 1, 2))
SIGN = ((1, -1, -1), (1, 1, 1), (1, -1, 1), (1, 1, 1), (-1, 1, 1), (-1, -1, 1))


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def _level(name, order, nr, na, limiter=3, roe=False, gravity=False, fallback=0, steps=1, cloud=False, graph=False):
    return {"name": name, "kind": "level", "order": order, "nr": nr, "na": na, "limiter": limiter, "roe": roe,
            "gravity": gravity, "fallback": fallback, "steps": steps, "cloud": cloud, "graph": graph}


def listed():
    return [
        # one step of the plain uniform solve (PLM-MC + Rusanov): launches and latency count
        _level("o2_step_32", 2, 32, 32),
        # the same solve as it is run in earnest: a CUDA graph of ten steps
        _level("o2_graph_32", 2, 32, 32, steps=10, graph=True),
        # the largest served second-order grid, here with Roe, minmod and gravity, after a cloud's insertion
        _level("o2_roe_96x64", 2, 96, 64, limiter=1, roe=True, gravity=True, steps=2, cloud=True),
        # a driver that owns its boxes: the second-order operator and its face fluxes on one ragged box
        {"name": "o2_box_45x37x31", "kind": "box", "order": 2, "nr": 64, "na": 64, "n0": 45, "n1": 37, "n2": 31,
         "limiter": 3, "roe": False, "gravity": False, "fallback": 0, "cloud": True},
        # the coarsest grid of a convergence study at fourth order (WENOZ + Roe)
        _level("o4_step_16", 4, 16, 16, roe=True),
        # the fourth-order uniform solve: 64 x 64^2 per panel, perturbed wind
        _level("o4_step_64", 4, 64, 64, roe=True),
        # an odd grid with the Rusanov solver and the PLM fallback, after a cloud's insertion
        _level("o4_rusanov_45x33", 4, 45, 33, fallback=1, cloud=True),
        # a large single solve with gravity after a cloud's insertion
        _level("o4_large_192x96", 4, 192, 96, roe=True, gravity=True, cloud=True),
        # the per-box fourth-order operator of one AMR patch, with face fluxes for the registers
        {"name": "o4_box_32", "kind": "box", "order": 4, "nr": 64, "na": 64, "n0": 32, "n1": 32, "n2": 32,
         "limiter": 3, "roe": True, "gravity": False, "fallback": 0, "cloud": False},
        # one AMR level's operator: 300 uneven boxes of 8^3 to 32^3 in one batch
        {"name": "o4_amr_batch_300", "kind": "batch", "nr": 192, "na": 192, "boxes": 300, "layout": 1, "roe": True,
         "gravity": False, "fallback": 0, "cloud": True},
        # four served fourth-order solves of different grids in flight together
        {"name": "o4_ensemble_4", "kind": "ensemble", "members": "32x32,48x32,32x48,64x32", "roe": True,
         "gravity": False, "fallback": 0, "steps": 1, "cloud": True},
        # a whole two-level AMR step: a 32 x 32^2 shell and 192 fine boxes of 8^3
        {"name": "amr_step_32", "kind": "amr", "nr": 32, "na": 32, "box": 8, "boxes": 192, "roe": True,
         "gravity": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["o2", "o2", "o4", "o4", "o4", "box", "batch", "ensemble", "amr"])
    roe, gravity, cloud = rng.random() < 0.6, rng.random() < 0.4, rng.random() < 0.5
    fallback = int(rng.random() < 0.25)
    if kind == "o2":
        case = _level("", 2, _log_int(rng, 16, 128), _log_int(rng, 16, 96), rng.choice([0, 1, 3, 3]), roe, gravity, 0,
                      rng.choice([1, 1, 2, 4]), cloud, rng.random() < 0.3)
    if kind == "o4":
        case = _level("", 4, _log_int(rng, 16, 160), _log_int(rng, 16, 96), 3, roe, gravity, fallback, 1, cloud,
                      rng.random() < 0.2)
    if kind in ("o2", "o4"):
        del case["name"]
        return case
    if kind == "box":
        n0, n1, n2 = (_log_int(rng, 8, 64) for _ in range(3))
        return {"kind": "box", "order": rng.choice([2, 4]), "nr": 64, "na": 64, "n0": n0, "n1": n1, "n2": n2,
                "limiter": rng.choice([0, 1, 3]), "roe": roe, "gravity": False, "fallback": fallback, "cloud": cloud}
    if kind == "batch":
        return {"kind": "batch", "nr": 192, "na": 192, "boxes": _log_int(rng, 20, 400), "layout": rng.randrange(1000),
                "roe": roe, "gravity": gravity, "fallback": fallback, "cloud": cloud}
    if kind == "ensemble":
        sizes = [f"{rng.choice([32, 48, 64])}x{rng.choice([24, 32, 48])}" for _ in range(rng.randint(2, 5))]
        return {"kind": "ensemble", "members": ",".join(sizes), "roe": roe, "gravity": gravity, "fallback": fallback,
                "steps": 1, "cloud": cloud}
    return {"kind": "amr", "nr": rng.randint(24, 48), "na": rng.randint(24, 40), "box": 8,
            "boxes": _log_int(rng, 30, 200), "roe": roe, "gravity": gravity}


def _members(case):
    return [tuple(int(x) for x in m.split("x")) for m in case["members"].split(",")]


def _batch_layout(case):
    """(panel, lo, hi) of the batch's boxes: sides 8 .. 32, the shapes from
    the case alone."""
    rng = random.Random(case["layout"])
    out = []
    for _ in range(case["boxes"]):
        n = [rng.randint(8, 32) if rng.random() < 0.5 else rng.choice([8, 16, 24, 32]) for _ in range(3)]
        lo = [rng.randint(0, case["nr"] - n[0]), rng.randint(0, case["na"] - n[1]), rng.randint(0, case["na"] - n[2])]
        out.append((rng.randrange(6), lo, [lo[d] + n[d] - 1 for d in range(3)]))
    return out


def _amr_layout(case):
    """Fine boxes tiling panel interiors (the fine level refines by 2)."""
    s, nrf, naf = case["box"], 2 * case["nr"], 2 * case["na"]
    out = []
    for b in (1, 3, 0, 2, 4, 5):
        for k in range(8, naf - 8 - s + 1, s):
            for j in range(8, naf - 8 - s + 1, s):
                for i in range(10, nrf - 10 - s + 1, s):
                    out.append((b, (i, j, k), (i + s - 1, j + s - 1, k + s - 1)))
    return out[:case["boxes"]]


def _box(case):
    """The box of a `box` case, at the low radial end and clear of the panel edges where it fits."""
    n = (case["n0"], case["n1"], case["n2"])
    lo = (0, (case["na"] - n[1]) // 2, (case["na"] - n[2]) // 2)
    return 1, lo, tuple(lo[d] + n[d] - 1 for d in range(3))


def work(case):
    """One pass: each input read once and each output written once.  FP64
    operations of the schemes per cell and stage: second order about 1400
    with Rusanov and 3000 with Roe (three faces: limited slopes, two local
    fluxes, the dissipation), fourth order about 9000 and 13000 (WENOZ of
    both sides of eight components on three faces, dissipation, mapped
    fluxes) and 1300 for the stage preparation."""
    roe = case["roe"]
    f2, f4 = (3000 if roe else 1400), (13000 if roe else 9000)
    kind = case["kind"]
    if kind == "level":
        cells = 6 * case["nr"] * case["na"] ** 2
        per = 4 * (f2 if case["order"] == 2 else f4 + 1300)
        return {"bytes": 128 * cells, "flops": per * cells * case["steps"]}
    if kind == "ensemble":
        cells = sum(6 * nr * na ** 2 for nr, na in _members(case))
        return {"bytes": 128 * cells, "flops": 4 * (f4 + 1300) * cells * case["steps"]}
    if kind == "amr":
        cells = 6 * case["nr"] * case["na"] ** 2 + sum(np.prod([h - a + 1 for a, h in zip(lo, hi)])
                                                       for _, lo, hi in _amr_layout(case))
        return {"bytes": int(128 * cells), "flops": int(4 * (f4 + 1300) * cells)}
    boxes = [_box(case)] if kind == "box" else _batch_layout(case)
    order = case.get("order", 4)
    g = 2 if order == 2 else 5
    moved = flops = 0
    for _, lo, hi in boxes:
        n = [hi[d] - lo[d] + 1 for d in range(3)]
        cells = math.prod(n)
        faces = sum(cells // n[d] * (n[d] + 1) for d in range(3))
        moved += 64 * (math.prod(x + 2 * g for x in n) + cells + faces)
        flops += cells * (f2 if order == 2 else f4)
    return {"bytes": moved, "flops": flops}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _Wind:
    """The seeded fields at points (unit direction X [3, ...], radius r):
    Cartesian primitives rho, v, p, B."""

    def __init__(self, seed, cloud):
        rng = np.random.default_rng(seed)
        self.kv = rng.normal(size=(2, 4, 3)) * 2.0
        self.ph = rng.uniform(0, 2 * PI, (2, 4))
        self.cm = rng.normal(size=(2, 4)) * 0.25
        ax = rng.normal(size=(2, 3))
        self.axis = ax / np.linalg.norm(ax, axis=1)[:, None]
        self.pulse_r = R_IN * rng.uniform(1.5, 5.0)
        self.cloud = cloud
        self.cloud_r = R_IN * rng.uniform(1.8, 2.4)
        self.cloud_size = R_IN * rng.uniform(0.4, 0.7)
        self.cloud_rho = rng.uniform(2.0, 5.0)
        self.cloud_v = rng.uniform(600e5, 1100e5)

    def _curl(self, X, m):
        """A tangential field: surface curl of a sum of four modes."""
        g = torch.zeros_like(X)
        for q in range(4):
            k = self.kv[m, q]
            c = self.cm[m, q] * torch.cos(k[0] * X[0] + k[1] * X[1] + k[2] * X[2] + self.ph[m, q])
            for d in range(3):
                g[d] += k[d] * c
        return torch.stack([g[1] * X[2] - g[2] * X[1], g[2] * X[0] - g[0] * X[2], g[0] * X[1] - g[1] * X[0]])

    def primitives(self, X, r):
        X = X + torch.zeros_like(r)
        s = R_IN / r
        rho = 700 * MP * s ** 2 + torch.zeros_like(X[0])
        v = 400e5 * (X + 0.05 * self._curl(X, 0))
        d2 = sum((r * X[d] - self.pulse_r * self.axis[0, d]) ** 2 for d in range(3)) / (0.3 * R_IN) ** 2
        p = 1e-7 * s ** (2 * GAMMA) * (1 + 0.5 * torch.exp(-0.5 * d2))
        B = 5e-3 * s ** 2 * (torch.sign(X[2]) * X + 0.05 * self._curl(X, 1))
        if self.cloud:
            inside = sum((r * X[d] - self.cloud_r * self.axis[1, d]) ** 2 for d in range(3)) < self.cloud_size ** 2
            rho = torch.where(inside, self.cloud_rho * rho, rho)
            p = torch.where(inside, 3 * p, p)
            v = torch.where(inside, self.cloud_v * X, v)
        return rho, v, p, B


def _level_state(nr, na, seed, cloud):
    """JU [6][8][k][j][i]: J x conserved values at the cell centres."""
    m = _Metrics(nr, na)
    i, a = m.index(0, nr), m.index(0, na)
    r, vol = m.radial(i)["rhalf"], m.radial(i)["vol"]
    wind = _Wind(seed, cloud)
    out = []
    for b in range(6):
        X = m.centre(b, a, a)[..., :, 0].permute(2, 0, 1)[..., None]
        rho, v, p, B = wind.primitives(X, r)
        u = _conserved(rho, v, p, B)
        out.append(u * (m.face(b, 0, a, a)["det"][..., None] * vol))
    return torch.stack(out)


def _box_input(case, box, seed, order):
    """Primitives (order 2) or native conserved values (order 4) of a box
    with its ghost cells."""
    block, lo, hi = box
    g = 2 if order == 2 else 5
    m = _Metrics(case["nr"], case["na"])
    i, j, k = (m.index(lo[d] - g, hi[d] + 1 + g) for d in range(3))
    A = m.centre(block, j, k)
    rho, v, p, B = _Wind(seed, case["cloud"]).primitives(A[..., :, 0].permute(2, 0, 1)[..., None], m.radial(i)["rhalf"])
    if order == 2:
        return torch.cat([rho[None], v, p[None], B])
    Ai = torch.linalg.inv(A).permute(2, 3, 0, 1)[..., None]
    u = _conserved(rho, v, p, B)
    return torch.cat([u[:1], _matvec(Ai, u[1:4]), u[4:5], _matvec(Ai, u[5:8])])


def _conserved(rho, v, p, B):
    e = p / (GAMMA - 1) + 0.5 * rho * (v ** 2).sum(0) + (B ** 2).sum(0) / (8 * PI)
    return torch.cat([rho[None], rho * v, e[None], B])


def _shell(case, nr, na, order):
    return hc.Shell(hc.Params(nr=nr, na=na, spatial_order=order, limiter=case.get("limiter", 3),
                              riemann_solver=2 if case["roe"] else 1, sun_gravity=int(case["gravity"]),
                              berta_fallback_type=case.get("fallback", 0), cfl=CFL))


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("level", "ensemble"):
        grids = [(case["nr"], case["na"])] if kind == "level" else _members(case)
        order = case.get("order", 4)
        shells = [_shell(case, nr, na, order) for nr, na in grids]
        first = [_level_state(nr, na, seed + 1000 * q, case["cloud"]).reshape(-1) for q, (nr, na) in enumerate(grids)]
        s = {"case": case, "shells": shells, "first": first, "ju": [u.clone() for u in first],
             "time": [torch.zeros(1, dtype=torch.float64, device=u.device) for u in first]}
        if kind == "ensemble":
            s["ensemble"] = Ensemble(shells)
        elif case["graph"]:
            s["graph"] = shells[0].capture_advance(s["ju"][0], case["steps"], s["time"][0])
        else:
            shells[0].advance(s["ju"][0], 1, s["time"][0])  # a handle that has stepped before
        return s
    if kind == "amr":
        coarse, fine = _shell(case, case["nr"], case["na"], 4), _shell(case, 2 * case["nr"], 2 * case["na"], 4)
        boxes = _amr_layout(case)
        ju = _level_state(case["nr"], case["na"], seed, False)
        fine_ju = _level_state(2 * case["nr"], 2 * case["na"], seed, False)
        step = AmrStep(coarse, fine, boxes)
        step.load(ju.reshape(-1), [fine_ju[b, :, lo[2]:hi[2] + 1, lo[1]:hi[1] + 1, lo[0]:hi[0] + 1]
                                   for b, lo, hi in boxes])
        dt = 0.1 / float(coarse.inv_dt_max(ju.reshape(-1)))
        return {"case": case, "step": step, "dt": dt, "boxes": len(boxes)}
    order = case.get("order", 4)
    shell = _shell(case, case["nr"], case["na"], order)
    boxes = [_box(case)] if kind == "box" else _batch_layout(case)
    n = [[hi[d] - lo[d] + 1 for d in range(3)] for _, lo, hi in boxes]
    zeros = lambda c: torch.zeros(8 * c, dtype=torch.float64, device=_device())  # noqa: E731
    rhs = zeros(sum(math.prod(x) for x in n))
    flux = [zeros(sum(math.prod(x) // x[d] * (x[d] + 1) for x in n)) for d in range(3)]
    works, at, fat = [], 0, [0, 0, 0]
    for q, (b, lo, hi) in enumerate(boxes):
        cells = math.prod(n[q])
        fl = []
        for d in range(3):
            c = 8 * (cells // n[q][d] * (n[q][d] + 1))
            fl.append(flux[d][fat[d]:fat[d] + c])
            fat[d] += c
        u = _box_input(case, (b, lo, hi), seed + q, order).reshape(-1).contiguous()
        works.append((make_box(lo, hi, 2 if order == 2 else 5, b), u, rhs[at:at + 8 * cells], fl))
        at += 8 * cells
    s = {"case": case, "shell": shell, "works": works, "rhs": rhs, "flux": flux}
    if kind == "batch":
        s["batch"] = O4Batch(shell, works)
    return s


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind in ("level", "ensemble"):
        for ju, first, time in zip(state["ju"], state["first"], state["time"]):
            ju.copy_(first)
            time.zero_()
        if kind == "ensemble":
            state["ensemble"].advance(state["ju"], case["steps"], state["time"])
        elif case["graph"]:
            state["graph"].replay()
        else:
            state["shells"][0].advance(state["ju"][0], case["steps"], state["time"][0])
        return {"ju": state["ju"], "time": state["time"]}
    if kind == "amr":
        state["step"].step(state["dt"])
        return {"coarse": state["step"].state_c,
                "fine": torch.cat([state["step"].fine_state(q) for q in range(state["boxes"])])}
    state["rhs"].zero_()
    if kind == "batch":
        state["batch"].rhs()
    else:
        box, u, rhs, flux = state["works"][0]
        (state["shell"].box_rhs if case["order"] == 2 else state["shell"].box_rhs_o4)(box, u, rhs, flux)
    return {"rhs": state["rhs"], "flux": state["flux"]}


# ---------------------------------------------------------------------------
# The same outputs in plain torch, 64 bits: the published scheme written
# over whole arrays [component][k][j][i].
# ---------------------------------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    if kind in ("level", "ensemble"):
        grids = [(case["nr"], case["na"])] if kind == "level" else _members(case)
        solve = _Order2 if case.get("order", 4) == 2 else _Order4
        ju, time = [], []
        for q, (nr, na) in enumerate(grids):
            u = _level_state(nr, na, seed + 1000 * q, case["cloud"])
            lv = solve(case, nr, na)
            t = torch.zeros(1, dtype=torch.float64, device=u.device)
            for _ in range(case["steps"]):
                dt = CFL / lv.metrics.cfl_rate(u)
                u = lv.step(u, dt)
                t = t + dt
            ju.append(u.reshape(-1))
            time.append(t)
        return {"ju": ju, "time": time}
    if kind == "amr":  # its coarse-fine interpolation and registers have no short closed form
        return None
    order = case.get("order", 4)
    m = _Metrics(case["nr"], case["na"])
    rhs, flux = [], [[], [], []]
    for q, box in enumerate([_box(case)] if kind == "box" else _batch_layout(case)):
        u = _box_input(case, box, seed + q, order)
        if order == 2:
            k, fl = _order2_box(m, box[0], box[1], u, case)
        else:
            k, fl = _order4_box(m, box[0], box[1], u, case)
        rhs.append(k.reshape(-1))
        for d in range(3):
            flux[d].append(fl[d].reshape(-1))
    return {"rhs": torch.cat(rhs), "flux": [torch.cat(f) for f in flux]}


def _matvec(M, x):
    """M [3][3]..., x [3]...."""
    return torch.stack([M[r, 0] * x[0] + M[r, 1] * x[1] + M[r, 2] * x[2] for r in range(3)])


def _cross(a, b):
    return torch.stack([a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]])


def _cofactor(A, d):
    """Row d of adj A; A [..., 3, 3]."""
    t1, t2 = (d + 1) % 3, (d + 2) % 3
    return torch.linalg.cross(A[..., :, t1], A[..., :, t2])


def _basis(b, x1, x2):
    """Equiangular gnomonic basis (Xhat, dXhat/dxi1, dXhat/dxi2), [..., 3, 3]."""
    x1, x2 = torch.broadcast_tensors(x1, x2)
    ta, tb = torch.tan(-PI / 4 + PI / 2 * x1), torch.tan(-PI / 4 + PI / 2 * x2)
    rho = torch.sqrt(1 + ta * ta + tb * tb)
    da, db, r3 = PI / 2 * (1 + ta * ta), PI / 2 * (1 + tb * tb), rho ** 3
    q = (1 / rho, ta / rho, tb / rho)
    q1 = (-ta / r3 * da, (1 / rho - ta * ta / r3) * da, -ta * tb / r3 * da)
    q2 = (-tb / r3 * db, -ta * tb / r3 * db, (1 / rho - tb * tb / r3) * db)
    rows = [torch.stack([SIGN[b][k] * c[PERM[b][k]] for c in (q, q1, q2)], -1) for k in range(3)]
    return torch.stack(rows, -2)


def _panel_coords(b, X):
    q = [None] * 3
    for k in range(3):
        q[PERM[b][k]] = SIGN[b][k] * X[k]
    return (np.arctan2(q[1], q[0]) + PI / 4) / (PI / 2), (np.arctan2(q[2], q[0]) + PI / 4) / (PI / 2)


def _panel_of(X):
    """Panel that holds direction X (numpy [3, ...]); ties to the lowest."""
    q0 = np.stack([sum(SIGN[b][k] * X[k] for k in range(3) if PERM[b][k] == 0) for b in range(6)])
    return np.argmax(q0 >= q0.max(0) - 1e-12, axis=0)


class _Metrics:
    """Radial and angular metrics as exact averages (8-point Gauss)."""

    def __init__(self, nr, na):
        self.nr, self.na = nr, na
        self.dx = (1.0 / nr, 1.0 / na, 1.0 / na)
        self.dev = _device()
        x, w = np.polynomial.legendre.leggauss(8)
        self.x = torch.tensor(0.5 * (x + 1), device=self.dev)
        self.w = torch.tensor(0.5 * w, device=self.dev)
        self._kept = {}

    def index(self, lo, hi):
        return torch.arange(lo, hi, device=self.dev, dtype=torch.float64)

    def radial(self, i):
        rt = (R_OUT - R_IN) / math.expm1(STRETCH)
        at = lambda x: R_IN + rt * torch.expm1(STRETCH * x * self.dx[0])  # noqa: E731
        lo, hi = at(i), at(i + 1)
        return {"rhalf": at(i + 0.5), "vol": (hi ** 3 - lo ** 3) / 3 / self.dx[0], "dr": (hi - lo) / self.dx[0],
                "area": (lo ** 2, (hi ** 2 - lo ** 2) / self.dx[0] / 2)}

    def centre(self, b, j, k):
        """Cell-centre basis [k][j][3][3]."""
        h = self.dx[1]
        return _basis(b, (j[None, :] + 0.5) * h, (k[:, None] + 0.5) * h)

    def face(self, b, d, j, k):
        """Averages over the low face of direction d of cells (j, k) (d = 0:
        over the cell): det, detA [k][j][3][3], the normal; the point basis A."""
        key = (b, d, float(j[0]), len(j), float(k[0]), len(k))
        if key in self._kept:
            return self._kept[key]
        h, x, w = self.dx[1], self.x, self.w
        J, K = j[None, :, None, None], k[:, None, None, None]
        if d == 0:
            A, wt = _basis(b, (J + x[:, None]) * h, (K + x) * h), w[:, None] * w
            P = self.centre(b, j, k)
        elif d == 1:
            A, wt = _basis(b, J * h, (K + x) * h), w[None, :]
            P = _basis(b, j[None, :] * h, (k[:, None] + 0.5) * h)
        else:
            A, wt = _basis(b, (J + x) * h, K * h), w[None, :]
            P = _basis(b, (j[None, :] + 0.5) * h, k[:, None] * h)
        det = torch.linalg.det(A)
        out = {"det": (wt * det).sum((-1, -2)), "detA": ((wt * det)[..., None, None] * A).sum((-3, -4)),
               "n": (wt[..., None] * _cofactor(A, d)).sum((-2, -3)), "A": P}
        self._kept[key] = out
        return out

    def mean_basis(self, b, j, k):
        h, x, w = self.dx[1], self.x, self.w
        A = _basis(b, (j[None, :, None, None] + x[:, None]) * h, (k[:, None, None, None] + x) * h)
        return ((w[:, None] * w)[..., None, None] * A).sum((-3, -4))

    def cfl_rate(self, ju):
        """Largest sum over directions of (fast speed bound + |v|) / width."""
        i, a = self.index(0, self.nr), self.index(0, self.na)
        R = self.radial(i)
        best = torch.zeros(1, dtype=torch.float64, device=self.dev)
        for b in range(6):
            f = [self.face(b, d, a, a) for d in range(3)]
            u = ju[b]
            rho = (u[0] / f[0]["det"][..., None] / R["vol"]).clamp(min=RHO_FLOOR)
            inv = torch.linalg.inv(f[0]["detA"]).permute(2, 3, 0, 1)[..., None]
            v, B = _matvec(inv, u[1:4]) / R["vol"] / rho, _matvec(inv, u[5:8]) / R["vol"]
            cell = f[0]["A"].permute(2, 3, 0, 1)[..., None]
            e = u[4] / f[0]["det"][..., None] / R["vol"]
            p = (GAMMA - 1) * (e - 0.5 * rho * (_matvec(cell, v) ** 2).sum(0) - (_matvec(cell, B) ** 2).sum(0) / (8 * PI))
            p = p.clamp(min=0)
            rate = 0
            for d in range(3):
                A = f[d]["A"].permute(2, 3, 0, 1)[..., None]
                v2, b2 = (_matvec(A, v) ** 2).sum(0), (_matvec(A, B) ** 2).sum(0)
                norm = torch.linalg.norm(f[d]["n"], dim=-1)[..., None]
                width = R["dr"] * self.dx[0] if d == 0 else R["vol"] * f[d]["det"][..., None] * self.dx[1] / R["area"][1] / norm
                rate = rate + (torch.sqrt(GAMMA * p / rho + b2 / (4 * PI) / rho) + torch.sqrt(v2)) / width
            best = torch.maximum(best, rate.max())
        return best


def _wind_inner(r):
    """Inner radial boundary: density, radial speed and pressure."""
    s = R_IN / r
    return 700 * MP * s ** 2, 500e5, 1e-7 * s ** (2 * GAMMA)


# --- Riemann dissipation ----------------------------------------------------
def _rusanov(wl, wr):
    c, speed = [], 0
    for w in (wl, wr):
        b2 = (w[5:8] ** 2).sum(0)
        c.append(_conserved(w[0], w[1:4], w[4], w[5:8]))
        s = w[1].abs() + torch.sqrt((GAMMA * w[4] + b2 / (4 * PI)) / w[0])
        speed = s if len(c) == 1 else torch.maximum(speed, s)
    return speed * (c[1] - c[0])


def _roe(wl, wr):
    """|A| (U_R - U_L) of the eight-wave Roe solver in the face frame with its
    entropy fix and fan check; Rusanov where the check fails."""
    where, one = torch.where, torch.ones_like(wl[0])
    ul, ur = _conserved(wl[0], wl[1:4], wl[4], wl[5:8]), _conserved(wr[0], wr[1:4], wr[4], wr[5:8])
    good = (wl[0] > 0) & (wr[0] > 0) & (wl[4] > 0) & (wr[4] > 0)
    al2, ar2 = GAMMA * wl[4] / wl[0], GAMMA * wr[4] / wr[0]
    mean = 0.5 * (wl + wr)
    rho, v, B = mean[0], mean[1:4], mean[5:8]
    ptot = 0.5 * (wl[4] + (wl[5:8] ** 2).sum(0) / (8 * PI) + wr[4] + (wr[5:8] ** 2).sum(0) / (8 * PI))
    byz2 = B[1] ** 2 + B[2] ** 2
    mag = (B[0] ** 2 + byz2) / (8 * PI)
    kk = 0.5 * (v ** 2).sum(0)
    cc = torch.minimum(torch.maximum(GAMMA * (ptot - mag) / rho, torch.minimum(al2, ar2)), torch.maximum(al2, ar2))
    good &= (cc > 0) & torch.isfinite(cc)
    cc = where(good, cc, one)
    c = torch.sqrt(cc)
    bb = B[0] ** 2 / (4 * PI) / rho
    b = torch.sqrt(bb)
    small = byz2 < 1e-18
    hyz = torch.sqrt(where(small, one, byz2))
    hyy = where(small, one / math.sqrt(2), B[1] / hyz)
    hzz = where(small, one / math.sqrt(2), B[2] / hyz)
    szb = cc + 2 * mag / rho
    h = torch.sqrt((szb * szb - 4 * cc * bb).clamp(min=0))
    aas, aaf = 0.5 * (szb - h), 0.5 * (szb + h)
    aas = where(small, torch.minimum(bb, cc), torch.minimum(aas.clamp(min=0), cc))
    aaf = where(small, torch.maximum(bb, cc), torch.maximum(aaf, cc))
    af, as_ = torch.sqrt(aaf), torch.sqrt(aas)
    dfs = aaf - aas
    alf = torch.sqrt(((cc - aas) / dfs).clamp(min=0))
    als = torch.sqrt(((aaf - cc) / dfs).clamp(min=0))
    alf, als = where(cc - aas <= 0, 0 * one, alf), where(cc - aas <= 0, one, als)
    alf, als = where((cc - aas > 0) & (aaf - cc <= 0), one, alf), where((cc - aas > 0) & (aaf - cc <= 0), 0 * one, als)
    alf, als = where(dfs < 1e-8, one, alf), where(dfs < 1e-8, 0 * one, als)
    sih = where(B[0] >= 0, one, -one)
    eig = [v[0], v[0], v[0] + b, v[0] - b, v[0] + af, v[0] - af, v[0] + as_, v[0] - as_]
    eps = ENTROPY * (v.abs().sum(0) + af)
    sp, s2p = torch.sqrt(PI * rho), torch.sqrt(2 * PI * rho)
    z = 0 * one
    t1, t2 = math.sqrt(0.5), 0.5 / s2p
    # right eigenvectors of the primitive system, then left ones
    fast = lambda s: [rho * alf, s * alf * af, -s * als * as_ * hyy * sih, -s * als * as_ * hzz * sih, alf * rho * cc, z,  # noqa: E731
                      2 * als * sp * c * hyy, 2 * als * sp * c * hzz]
    slow = lambda s: [rho * als, s * als * as_, s * alf * af * hyy * sih, s * alf * af * hzz * sih, als * rho * cc, z,  # noqa: E731
                      -2 * alf * sp * c * hyy, -2 * alf * sp * c * hzz]
    alfven = lambda s: [z, z, -hzz * t1, hyy * t1, z, z, s * hzz * s2p * sih, -s * hyy * s2p * sih]  # noqa: E731
    right = [[one, z, z, z, z, z, z, z], [z, z, z, z, z, one, z, z], alfven(1), alfven(-1), fast(1), fast(-1), slow(1), slow(-1)]
    lfast = lambda s: [z, s * 0.5 * alf * af / cc, -s * 0.5 * als * as_ * hyy * sih / cc, -s * 0.5 * als * as_ * hzz * sih / cc,  # noqa: E731
                       0.5 * alf / (cc * rho), z, 0.25 * als * hyy / (c * sp), 0.25 * als * hzz / (c * sp)]
    lslow = lambda s: [z, s * 0.5 * als * as_ / cc, s * 0.5 * alf * af * hyy * sih / cc, s * 0.5 * alf * af * hzz * sih / cc,  # noqa: E731
                       0.5 * als / (cc * rho), z, -0.25 * alf * hyy / (c * sp), -0.25 * alf * hzz / (c * sp)]
    lalf = lambda s: [z, z, -hzz * t1, hyy * t1, z, z, s * hzz * sih * t2, -s * hyy * sih * t2]  # noqa: E731
    left = [[one, z, z, z, -1 / cc, z, z, z], [z, z, z, z, z, one, z, z], lalf(1), lalf(-1), lfast(1), lfast(-1), lslow(1), lslow(-1)]
    dc = ul - ur
    dp = (GAMMA - 1) * (kk * dc[0] - (v * dc[1:4]).sum(0) + dc[4] - (B * dc[5:8]).sum(0) / (4 * PI))
    du = torch.cat([dc[:1], (dc[1:4] - v * dc[0]) / rho, dp[None], dc[5:8]])
    al = [sum(left[k][q] * du[q] for q in range(8)) for k in range(8)]

    def to_conserved(d):
        d = torch.stack(d)
        return torch.cat([d[:1], v * d[0] + rho * d[1:4],
                          (kk * d[0] + rho * (v * d[1:4]).sum(0) + d[4] / (GAMMA - 1) + (B * d[5:8]).sum(0) / (4 * PI))[None],
                          d[5:8]])

    state, order = ul, (5, 3, 7, 0, 1, 6, 2, 4)
    for q in range(7):
        k = order[q]
        state = state - to_conserved([al[k] * x for x in right[k]])
        thermal = state[4] - 0.5 * (state[1:4] ** 2).sum(0) / state[0] - (state[5:8] ** 2).sum(0) / (8 * PI)
        fine = (state[0] > 0) & torch.isfinite(state[0]) & (thermal >= 0) & torch.isfinite(thermal)
        good &= fine | ~(eig[order[q + 1]] > eig[k])
    lu = [where(e.abs() >= eps, e.abs(), 0.5 * (e * e + eps * eps) / eps) * a for e, a in zip(eig, al)]
    out = -to_conserved([sum(right[k][r] * lu[k] for k in range(8)) for r in range(8)])
    good &= torch.isfinite(out).all(0)
    return where(good, out, _rusanov(wl, wr))


# --- second order -----------------------------------------------------------
def _primitives(u):
    rho = u[0].clamp(min=RHO_FLOOR)
    v = u[1:4] / rho
    p = (GAMMA - 1) * (u[4] - 0.5 * rho * (v ** 2).sum(0) - (u[5:8] ** 2).sum(0) / (8 * PI))
    return torch.cat([rho[None], v, p.clamp(min=0)[None], u[5:8]])


def _slope(a, b, limiter):
    """Limited slope of the differences a, b on both sides of a cell."""
    if limiter == 0:
        return 0.5 * (a + b)
    m = torch.where(a > 0, torch.minimum(a, b), torch.maximum(a, b))
    if limiter == 3:
        m = torch.sign(a) * torch.minimum(0.5 * (a + b).abs(), 2 * torch.minimum(a.abs(), b.abs()))
    return torch.where(a * b <= 0, torch.zeros_like(a), m)


def _face_states(w, d, limiter):
    """Left and right states of the faces of direction d; w has two ghost layers."""
    ax = 3 - d
    for q in range(3):
        if q != d:
            w = w.narrow(3 - q, 2, w.shape[3 - q] - 4)
    n = w.shape[ax] - 3
    mm, m, c, p = (w.narrow(ax, s, n) for s in range(4))
    l = m + 0.5 * _slope(m - mm, c - m, limiter)
    r = c - 0.5 * _slope(c - m, p - c, limiter)
    l = torch.where((l[0] >= RHO_FLOOR) & (l[4] >= 0), l, m)
    r = torch.where((r[0] >= RHO_FLOOR) & (r[4] >= 0), r, c)
    return l, r


def _frame(n):
    """Rows: unit normal, two tangents; n [3][k][j]."""
    norm = torch.sqrt((n ** 2).sum(0))
    f0 = n / norm
    axis = (f0.abs() <= f0.abs().min(0).values + 1e-12).to(torch.int64).argmax(0)  # least aligned, first of ties
    f1 = torch.zeros_like(f0)
    for a in range(3):
        t = torch.zeros_like(f0)
        t[(a + 1) % 3], t[(a + 2) % 3] = f0[(a + 2) % 3], -f0[(a + 1) % 3]
        f1 = torch.where(axis == a, t, f1)
    f1 = f1 / torch.sqrt((f1 ** 2).sum(0))
    return torch.stack([f0, f1, _cross(f0, f1)]), norm


def _order2_flux(l, r, n, area, roe):
    f, norm = _frame(n.permute(2, 0, 1))
    f = f[..., None]
    loc, flux = [], 0
    for s in (l, r):
        q = torch.cat([s[:1], _matvec(f, s[1:4]), s[4:5], _matvec(f, s[5:8])])
        pt = q[4] + (q[5:8] ** 2).sum(0) / (8 * PI)
        u = _conserved(q[0], q[1:4], q[4], q[5:8])
        g = torch.cat([(q[0] * q[1])[None], q[0] * q[1] * q[1:4] - q[5] * q[5:8] / (4 * PI),
                       ((u[4] + pt) * q[1] - q[5] * (q[1:4] * q[5:8]).sum(0) / (4 * PI))[None], q[1] * q[5:8] - q[1:4] * q[5]])
        g[1] += pt
        loc.append(q)
        flux = flux + g
    num = 0.5 * area * norm[..., None] * (flux - (_roe if roe else _rusanov)(*loc))
    ft = f.transpose(0, 1)
    return torch.cat([num[:1], _matvec(ft, num[1:4]), num[4:5], _matvec(ft, num[5:8])])


def _order2_rhs(m, block, lo, w, case, states):
    """rhs and fluxes of one box from the face states of its directions."""
    n = [w.shape[3 - d] - 4 for d in range(3)]
    idx = [m.index(lo[d], lo[d] + n[d] + 1) for d in range(3)]
    wv = w[:, 2:-2, 2:-2, 2:-2]
    rhs, md, fluxes = torch.zeros_like(wv), 0, []
    if case["gravity"]:
        f = m.face(block, 0, idx[1][:-1], idx[2][:-1])
        q = -GM * m.radial(idx[0][:-1])["dr"] * wv[0]
        X = f["A"][..., :, 0].permute(2, 0, 1)[..., None]
        rhs[1:4] += q * f["detA"][..., :, 0].permute(2, 0, 1)[..., None]
        rhs[4] += q * f["det"][..., None] * (X * wv[1:4]).sum(0)
    for d in range(3):
        l, r = states[d]
        j, k = (idx[1] if d == 1 else idx[1][:-1]), (idx[2] if d == 2 else idx[2][:-1])
        nrm = m.face(block, d, j, k)["n"]
        area = m.radial(idx[0] if d == 0 else idx[0][:-1])["area"][min(d, 1)]
        F = _order2_flux(l, r, nrm, area, case["roe"])
        fluxes.append(F)
        bf = (0.5 * (l[5:8] + r[5:8]) * nrm.permute(2, 0, 1)[..., None]).sum(0) * area
        rhs -= torch.diff(F, dim=3 - d) / m.dx[d]
        md = md - torch.diff(bf, dim=2 - d) / m.dx[d]
    rhs[1:4] += md * wv[5:8] / (4 * PI)
    rhs[5:8] += md * wv[1:4]
    rhs[4] += md * (wv[1:4] * wv[5:8]).sum(0) / (4 * PI)
    return rhs, fluxes


def _order2_box(m, block, lo, w, case):
    return _order2_rhs(m, block, lo, w, dict(case, gravity=False), [_face_states(w, d, case["limiter"]) for d in range(3)])


def _edge(b, ax, side, na):
    """Adjacent panel across an edge, its axis and side, and the adjacent
    along-edge index of each along-edge cell."""
    h = 1.0 / na
    t = (np.arange(na) + 0.5) * h

    def coords(e, s):
        A = _basis(b, *(torch.as_tensor(v, dtype=torch.float64) for v in ((e, s) if ax == 1 else (s, e))))
        return A[..., :, 0].movedim(-1, 0).numpy()

    X = coords(-0.5 * h if side == 0 else 1 + 0.5 * h, 0.5)
    nb = int(_panel_of(X))
    y1, y2 = _panel_coords(nb, X)
    nax = 1 if min(y1, 1 - y1) < min(y2, 1 - y2) else 2
    nside = 0 if (y1 if nax == 1 else y2) < 0.5 else 1
    y = _panel_coords(nb, coords(float(side), t))
    return nb, nax, nside, np.rint(y[2 - nax] / h - 0.5).astype(int)


class _Order2:
    """The second-order level: primitives with ghosts, shared seam states."""

    def __init__(self, case, nr, na):
        self.case, self.metrics, self.nr, self.na = case, _Metrics(nr, na), nr, na
        m, h = self.metrics, 1.0 / na
        a = m.index(0, na)
        self.vol = m.radial(m.index(0, nr))["vol"]
        self.det = torch.stack([m.face(b, 0, a, a)["det"] for b in range(6)])
        self.edges = {(b, ax, s): _edge(b, ax, s, na) for b in range(6) for ax in (1, 2) for s in (0, 1)}
        self.donors = {}
        for (b, ax, side), (nb, nax, nside, _) in self.edges.items():
            for g in range(2):
                e = torch.tensor(-(g + 0.5) * h if side == 0 else 1 + (g + 0.5) * h, dtype=torch.float64)
                t = torch.tensor((np.arange(na) + 0.5) * h)
                A = _basis(b, e, t) if ax == 1 else _basis(b, t, e)
                y = _panel_coords(nb, A[..., :, 0].movedim(-1, 0).numpy())
                u = y[2 - nax] / h - 0.5
                base = np.clip(np.floor(u).astype(int) - 1, 0, na - 4)
                wt = np.ones((4, na))
                for q in range(4):
                    for r in range(4):
                        if r != q:
                            wt[q] *= (u - (base + r)) / (q - r)
                self.donors[b, ax, side, g] = (nb, nax, g if nside == 0 else na - 1 - g,
                                               torch.tensor(base, device=m.dev), torch.tensor(wt, device=m.dev))

    def prepare(self, ju):
        m, nr, na = self.metrics, self.nr, self.na
        w = torch.zeros((6, 8, na + 4, na + 4, nr + 4), dtype=torch.float64, device=m.dev)
        v = torch.stack([_primitives(ju[b] / (self.vol * self.det[b][..., None])) for b in range(6)])
        w[:, :, 2:-2, 2:-2, 2:-2] = v
        for (b, ax, side, g), (nb, nax, layer, base, wt) in self.donors.items():
            row = v[nb][:, :, layer] if nax == 1 else v[nb][:, layer]
            x = sum(wt[q][:, None] * row[:, base + q] for q in range(4))
            x[0].clamp_(min=RHO_FLOOR)
            x[4].clamp_(min=0)
            at = 1 - g if side == 0 else na + 2 + g
            (w[b][:, 2:-2, at] if ax == 1 else w[b][:, at, 2:-2])[..., 2:-2] = x
        a = m.index(0, na)
        rl = m.radial(m.index(nr - 1, nr))["rhalf"]
        for b in range(6):
            A = m.centre(b, a, a).permute(2, 3, 0, 1)
            Ai = torch.linalg.inv(m.centre(b, a, a)).permute(2, 3, 0, 1)
            for g in range(2):
                rho, ur, p = _wind_inner(m.radial(m.index(g - 2, g - 1))["rhalf"])
                inner = w[b][:, 2:-2, 2:-2, g]
                inner[0], inner[1:4], inner[4], inner[5:8] = rho, ur * A[:, 0], p, 0
            last = v[b][..., -1]
            u = _conserved(last[0], last[1:4], last[4], last[5:8])
            u = torch.cat([u[:1], _matvec(Ai, u[1:4]), u[4:5], _matvec(Ai, u[5:8])])
            for g in range(2):
                s = rl / m.radial(m.index(nr + g, nr + g + 1))["rhalf"]
                ug = torch.cat([u[:6] * s ** 2, u[6:] * s])
                w[b][:, 2:-2, 2:-2, nr + 2 + g] = _primitives(torch.cat([ug[:1], _matvec(A, ug[1:4]), ug[4:5], _matvec(A, ug[5:8])]))
        return w

    def rhs(self, w):
        own = [[list(_face_states(w[b], d, self.case["limiter"])) for d in range(3)] for b in range(6)]
        shared = [[[x.clone() for x in own[b][d]] for d in range(3)] for b in range(6)]
        for (b, ax, side), (nb, nax, nside, along) in self.edges.items():
            src = own[nb][nax][1 if nside == 0 else 0]
            slab = src[:, :, 0 if nside == 0 else -1] if nax == 1 else src[:, 0 if nside == 0 else -1]
            dst = shared[b][ax][0 if side == 0 else 1]
            (dst[:, :, 0 if side == 0 else -1] if ax == 1 else dst[:, 0 if side == 0 else -1])[:] = slab[:, torch.as_tensor(along, device=slab.device)]
        return torch.stack([_order2_rhs(self.metrics, b, (0, 0, 0), w[b], self.case, shared[b])[0] for b in range(6)])

    def step(self, u, dt):
        return _rk4(u, dt, lambda x, weight: self.rhs(self.prepare(x)))


def _rk4(u, dt, rhs):
    out, x = u, u
    for b, a in ((1 / 6, 0.5), (1 / 3, 0.5), (1 / 3, 1.0), (1 / 6, None)):
        k = rhs(x, dt * b)
        out = out + dt * b * k
        x = u + dt * a * k if a else None
    return out


# --- fourth order -----------------------------------------------------------
def _at(x, d, s):
    """x at index + s along direction d (i, j, k = last axes); wraps, and the
    wrapped cells are never part of a result."""
    return torch.roll(x, -s, -1 - d)


def _diff(x, d):
    return 0.5 * _at(x, d, 1) - 0.5 * _at(x, d, -1)


def _lap(x, dirs):
    return sum(_at(x, d, 1) + _at(x, d, -1) - 2 * x for d in dirs)


def _product(a, b, dirs):
    """Fourth-order average of a product from averages."""
    return a * b + sum(_diff(a, d) * _diff(b, d) for d in dirs) / 12


def _native_primitives(u, A):
    rho = u[0].clamp(min=RHO_FLOOR)
    v = u[1:4] / rho
    ke, me = 0.5 * rho * (_matvec(A, v) ** 2).sum(0), (_matvec(A, u[5:8]) ** 2).sum(0) / (8 * PI)
    p = ((u[4] - ke - me) * (GAMMA - 1)).clamp(min=0)
    return torch.cat([rho[None], v, p[None], u[5:8]])


def _normalised(v):
    scale = torch.stack([x.abs() for x in v]).max(0).values
    inv = torch.where(scale > 0, 1 / scale, scale)
    return [x * inv for x in v], scale


def _wenoz(v):
    """Left and right states from six cells, both sides of each face."""
    v, scale = _normalised(v)
    out = []
    for a, b, c, d, e in ((v[0], v[1], v[2], v[3], v[4]), (v[5], v[4], v[3], v[2], v[1])):
        q = ((3 * a - 10 * b + 15 * c) / 8, (-b + 6 * c + 3 * d) / 8, (3 * c + 6 * d - e) / 8)
        beta = (13 / 12 * (a - 2 * b + c) ** 2 + (a - 4 * b + 3 * c) ** 2 / 4,
                13 / 12 * (b - 2 * c + d) ** 2 + (b - d) ** 2 / 4,
                13 / 12 * (c - 2 * d + e) ** 2 + (3 * c - 4 * d + e) ** 2 / 4)
        tau = (beta[0] - beta[2]).abs()
        al = [w * (1 + tau / (x + 1e-40)) for w, x in zip((1 / 16, 5 / 8, 5 / 16), beta)]
        out.append(scale * (al[0] * q[0] + al[1] * q[1] + al[2] * q[2]) / (al[0] + al[1] + al[2]))
    return out


def _weno3(v, eps):
    v, scale = _normalised(v)
    out = []
    for a, b, c in ((v[0], v[1], v[2]), (v[3], v[2], v[1])):
        dm, dp = b - a, c - b
        tau = (dp - dm) ** 2
        w0, w1 = 0.75 * (1 + tau / (dp * dp + eps)), 0.25 * (1 + tau / (dm * dm + eps))
        out.append(scale * (w0 * 0.5 * (b + c) + w1 * 0.5 * (3 * b - a)) / (w0 + w1))
    return out


def _minmod3(a, b, c):
    lo, hi = torch.minimum(a, torch.minimum(b, c)), torch.maximum(a, torch.maximum(b, c))
    return torch.where(lo > 0, lo, torch.where(hi < 0, hi, torch.zeros_like(a)))


def _plm(v):
    l = v[1] + 0.5 * _minmod3(1.5 * (v[1] - v[0]), 0.5 * (v[2] - v[0]), 1.5 * (v[2] - v[1]))
    r = v[2] - 0.5 * _minmod3(1.5 * (v[2] - v[1]), 0.5 * (v[3] - v[1]), 1.5 * (v[3] - v[2]))
    return l, r


def _order4_box(m, block, lo, U, case):
    """rhs and face fluxes of one box; U native averages with five ghost layers."""
    n = [U.shape[-1 - d] - 10 for d in range(3)]
    i, j, k = (m.index(lo[d] - 5, lo[d] + n[d] + 5) for d in range(3))
    R = m.radial(i)
    put = lambda x: x.movedim((-2, -1), (0, 1))[..., None] if x.dim() == 4 else x.movedim(-1, 0)[..., None]  # noqa: E731
    A0 = put(m.centre(block, j, k))

    def within(x, g):
        y = torch.zeros_like(x)
        s = slice(g, -g)
        y[..., s, s, s] = x[..., s, s, s]
        return y

    # detector, point values
    WA = _native_primitives(U, A0)
    sens = (WA[0], WA[4], 0.5 * (WA[5:8] ** 2).sum(0))
    eta2 = 0
    for d in range(3):
        e = torch.stack([(_at(q, d, 1) - 2 * q + _at(q, d, -1)).abs() /
                         (_at(q, d, 1).abs() + 2 * q.abs() + _at(q, d, -1).abs() + 1e-40) for q in sens])
        eta2 = eta2 + e.max(0).values ** 2
    raw = within((torch.sqrt(eta2) < ETA_D).to(torch.float64), 1)
    th = raw
    for d in range(3):
        th = torch.minimum(th, torch.minimum(_at(raw, d, 1), _at(raw, d, -1)))
    th = within(th, 2)
    WP = _native_primitives(torch.where(th > 0.5, U - _lap(U, range(3)) / 24, U), A0)

    rhs, mj, fluxes = torch.zeros_like(U), 0, []
    for d in range(3):
        tr = [t for t in range(3) if t != d]
        f = m.face(block, d, j, k)
        det, detA, nrm, A = f["det"][..., None], put(f["detA"]), put(f["n"]), put(f["A"])
        area = R["area"][min(d, 1)]
        cells = [_at(WP, d, s) for s in range(-3, 3)]
        smooth = torch.stack([_at(th, d, s) for s in range(-3, 3)]).min(0).values > 0.5
        thf = torch.minimum(_at(th, d, -1), th)
        fb = _plm(cells[1:5]) if case["fallback"] else _weno3(cells[1:5], m.dx[d] ** 2)
        l, r = (torch.where(smooth, w, q) for w, q in zip(_wenoz(cells), fb))
        for s in (l, r):
            s[0].clamp_(min=RHO_FLOOR)
            s[4].clamp_(min=1e-12)
        if case["roe"]:
            usable = lambda w: torch.isfinite(w).all(0) & (w[0] >= RHO_FLOOR) & (w[4] >= 0)  # noqa: E731
            cl, cr = _at(WA, d, -1), WA
            fix = ~(usable(l) & usable(r)) & usable(cl) & usable(cr)
            l, r, thf = torch.where(fix, cl, l), torch.where(fix, cr, r), torch.where(fix, 0 * thf, thf)
        fs, ps, phys = 0, 0, []
        for s in (l, r):
            vc, bc = _matvec(A, s[1:4]), _matvec(A, s[5:8])
            ke, me, vb = 0.5 * s[0] * (vc ** 2).sum(0), (bc ** 2).sum(0) / (8 * PI), (vc * bc).sum(0)
            vn, bn = s[1 + d], s[5 + d]
            fs = fs + torch.cat([(s[0] * vn)[None], s[0] * vn * s[1:4] - bn * s[5:8] / (4 * PI),
                                 ((2 * me + ke + s[4] * GAMMA / (GAMMA - 1)) * vn - bn * vb / (4 * PI))[None],
                                 vn * s[5:8] - s[1:4] * bn])
            ps = ps + s[4] + me
            phys.append((torch.cat([s[:1], vc, s[4:5], bc]), ke + me + s[4] / (GAMMA - 1)))
        apoint = area if d == 0 else area - _lap(area, [0]) / 24
        if case["roe"]:
            frame = [torch.linalg.cross(f["A"][..., :, (d + 1) % 3], f["A"][..., :, (d + 2) % 3]), f["A"][..., :, (d + 1) % 3]]
            size = torch.linalg.norm(frame[0], dim=-1)[..., None]
            frame = [put(x / torch.linalg.norm(x, dim=-1, keepdim=True)) for x in frame]
            F = torch.stack([*frame, _cross(*frame)])
            loc = [torch.cat([q[:1].clamp(min=RHO_FLOOR), _matvec(F, q[1:4]), q[4:5].clamp(min=0), _matvec(F, q[5:8])]) for q, _ in phys]
            q = apoint * size * _roe(*loc)
            inv, dt = put(torch.linalg.inv(f["A"])), torch.linalg.det(f["A"])[..., None]
            Ft = F.transpose(0, 1)
            qd = torch.cat([q[:1], _matvec(inv, _matvec(Ft, q[1:4])), q[4:5], _matvec(inv, _matvec(Ft, q[5:8]))]) / dt
        else:
            cons = [torch.cat([s[:1], s[0] * s[1:4], e[None], s[5:8]]) for s, (_, e) in zip((l, r), phys)]
            qd = apoint * cons[1] - apoint * cons[0]
        sm = thf > 0.5
        average = lambda x: torch.where(sm, x + _lap(x, tr) / 24, x)  # noqa: E731
        fa, pa = average(fs), average(ps)

        def mapped(x, y):
            """det or detA times the averages x, transverse corrections from y."""
            prod = lambda g, c: g * x[c] + sum(_diff(g, t) * _diff(y[c], t) for t in tr) / 12  # noqa: E731
            D = det + 0 * x[0]
            M = detA + 0 * x[0]
            vec = lambda s: torch.stack([sum(prod(M[a, c], s + c) for c in range(3)) for a in range(3)])  # noqa: E731
            return torch.cat([prod(D, 0)[None], vec(1), prod(D, 4)[None], vec(5)])

        flux = _product(mapped(fa, fa), area + 0 * pa, tr)
        t3 = _product(pa, area + 0 * pa, tr)
        flux[1:4] += torch.stack([_product(x + 0 * t3, t3, tr) for x in nrm])
        if case["roe"]:
            diss = mapped(average(qd), qd)
        else:
            qv = average(qd)
            s = 0.5 * (l + r)
            p, rho = s[4].clamp(min=0), s[0].clamp(min=RHO_FLOOR)
            bc = _matvec(A, s[5:8])
            bm, bn = torch.sqrt((bc ** 2).sum(0)), (A[:, 0] * bc).sum(0)
            ce = torch.sqrt(GAMMA * p / rho)
            aa, cross = ce * ce + bm * bm / (4 * PI * rho), bn.abs() * ce / torch.sqrt(PI * rho)
            fast = 0.5 * (torch.sqrt((aa + cross).clamp(min=0)) + torch.sqrt((aa - cross).clamp(min=0)))
            speed = s[1 + d].abs() + fast * torch.sqrt((A[:, d] ** 2).sum(0))
            diss = speed * torch.cat([(det * qv[0])[None], _matvec(detA, qv[1:4]), (det * qv[4])[None], _matvec(detA, qv[5:8])])
        fx = 0.5 * (flux - diss)
        fluxes.append(fx)
        rhs -= (_at(fx, d, 1) - fx) / m.dx[d]
        # normal field of the Powell term
        u = U[5 + d]
        bface = 7 / 12 * (_at(u, d, -1) + u) - 1 / 12 * (_at(u, d, -2) + _at(u, d, 1))
        bf = torch.where(thf <= 0.5, det * 0.5 * (l[5 + d] + r[5 + d]), _product(det + 0 * u, bface, tr))
        bp = _product(bf, area + 0 * u, tr)
        mj = mj - (_at(bp, d, 1) - bp) / m.dx[d]
    vel, mag = _matvec(A0, WP[1:4]), _matvec(A0, WP[5:8]) / (4 * PI)
    K = torch.cat([torch.zeros_like(mj)[None], mag, (vel * mag).sum(0)[None], vel])
    rhs += _product(mj, K + _lap(K, range(3)) / 24, range(3))
    if case["gravity"]:
        f = m.face(block, 0, j, k)
        dr = R["dr"] + 0 * U[0]
        rd, re = _product(dr, U[0], [0]), _product(dr, U[1], [0])
        col = put(f["detA"])[:, 0]
        rhs[1:4] -= GM * torch.stack([_product(x + 0 * rd, rd, (1, 2)) for x in col])
        rhs[4] -= GM * _product(f["det"][..., None] + 0 * re, re, (1, 2))
    valid = [slice(5, 5 + n[d]) for d in (2, 1, 0)]
    cut = lambda d: [slice(5, 5 + n[q] + (q == d)) for q in (2, 1, 0)]  # noqa: E731
    return rhs[(slice(None), *valid)], [fluxes[d][(slice(None), *cut(d))] for d in range(3)]


def _one_sided(x, ax):
    """Undivided centred difference; second-order one-sided at both ends."""
    n = x.shape[ax]
    s = lambda q: x.narrow(ax, q, 1)  # noqa: E731
    mid = 0.5 * x.narrow(ax, 2, n - 2) - 0.5 * x.narrow(ax, 0, n - 2)
    return torch.cat([-1.5 * s(0) + 2 * s(1) - 0.5 * s(2), mid, 0.5 * s(n - 3) - 2 * s(n - 2) + 1.5 * s(n - 1)], ax)


def _average_weights(u, base):
    """Weights of four cell averages base .. base + 3 for the point value at
    u of the cubic that matches them."""
    w = np.zeros((4, len(u)))
    dl = np.zeros((5, len(u)), dtype=np.longdouble)
    for n in range(5):
        for r in range(5):
            if r == n:
                continue
            t = np.full(len(u), 1, dtype=np.longdouble) / (n - r)
            for q in range(5):
                if q not in (n, r):
                    t *= (u - (base + q)) / np.longdouble(n - q)
            dl[n] += t
    for q in range(4):
        w[q] = dl[q + 1:].sum(0)
    return w


class _Order4:
    """The fourth-order level: Cartesian averages with seam ghosts, native
    averages, the operator per panel, seam fluxes reconciled after the step."""

    GA = 6  # angular ghost layers of the Cartesian averages

    def __init__(self, case, nr, na):
        self.case, self.metrics, self.nr, self.na = case, _Metrics(nr, na), nr, na
        m, g, h = self.metrics, self.GA, 1.0 / na
        self.edges = {(b, ax, s): _edge(b, ax, s, na) for b in range(6) for ax in (1, 2) for s in (0, 1)}
        idx = np.arange(-g - 1, na + g + 1)
        kk, jj = np.meshgrid(idx, idx, indexing="ij")
        need = ~((jj >= 1) & (jj < na - 1) & (kk >= 1) & (kk < na - 1))
        self.need = torch.tensor(need, device=m.dev)
        pj, pk = jj[need], kk[need]
        self.points = []
        for b in range(6):
            A = _basis(b, torch.tensor((pj + 0.5) * h), torch.tensor((pk + 0.5) * h))
            X = A[:, :, 0].T.numpy()
            p = _panel_of(X)
            y = np.zeros((2, len(p)))
            for q in range(6):
                y[:, p == q] = _panel_coords(q, X[:, p == q])
            u = y.astype(np.longdouble) / h
            base = np.clip(np.floor(u.astype(float)).astype(int) - 1, 0, na - 4)
            cell = np.clip(np.floor(u.astype(float)).astype(int), 0, na - 1)
            t = lambda x: torch.tensor(np.ascontiguousarray(x), device=m.dev)  # noqa: E731
            self.points.append((t(p), t(base), t(cell), t(_average_weights(u[0], base[0])), t(_average_weights(u[1], base[1]))))
        e = m.index(-g, na + g)
        self.meanA = [m.mean_basis(b, e, e) for b in range(6)]
        ext = m.index(-1, na + 1)
        self.det = [m.face(b, 0, ext, ext)["det"] for b in range(6)]

    def cartesian(self, ju):
        m, nr, na, g = self.metrics, self.nr, self.na, self.GA
        vol = m.radial(m.index(-1, nr + 1))["vol"]
        dvol, vol = 0.5 * (vol[2:] - vol[:-2]), vol[1:-1]
        C = torch.zeros((6, 8, na + 2 * g, na + 2 * g, nr), dtype=torch.float64, device=m.dev)
        for b in range(6):
            D = self.det[b]
            det = D[1:-1, 1:-1, None]
            q = ju[b] / det
            d1, d2 = 0.5 * (D[1:-1, 2:] - D[1:-1, :-2])[..., None], 0.5 * (D[2:, 1:-1] - D[:-2, 1:-1])[..., None]
            ang = (ju[b] - (_one_sided(q, 2) * d1 + _one_sided(q, 1) * d2) / 12) / det
            C[b][:, g:-g, g:-g] = (ang - _one_sided(ang / vol, 3) * dvol / 12) / vol
        V = C[:, :, g:-g, g:-g].clone()
        for b in range(6):
            p, base, cell, wj, wk = self.points[b]
            pts = 0
            for s in range(4):
                for q in range(4):
                    pts = pts + (wk[s] * wj[q])[:, None, None] * V[p, :, base[1] + s, base[0] + q]
            grid = torch.zeros((8, na + 2 * g + 2, na + 2 * g + 2, nr), dtype=torch.float64, device=m.dev)
            grid[:, self.need] = pts.transpose(0, 1)
            own = torch.zeros_like(grid)
            own[:, self.need] = V[p, :, cell[1], cell[0]].transpose(0, 1)
            own = own[:, 1:-1, 1:-1]
            u = 5 / 6 * grid + (_lap(grid, (1, 2)) + 4 * grid) / 24
            u = u[:, 1:-1, 1:-1]
            thermal = u[4] - torch.where(u[0] > 0, 0.5 * (u[1:4] ** 2).sum(0) / u[0] + (u[5:8] ** 2).sum(0) / (8 * PI), 0 * u[0])
            ok = torch.isfinite(u).all(0) & (u[0] >= RHO_FLOOR) & (thermal >= 0)
            u = torch.where(ok, u, own)
            u[:, g:-g, g:-g] = V[b]
            C[b] = u
        return C

    def prepare(self, ju):
        m, nr, na, g = self.metrics, self.nr, self.na, self.GA
        C = self.cartesian(ju)
        out = torch.zeros((6, 8, na + 10, na + 10, nr + 10), dtype=torch.float64, device=m.dev)
        e, s = m.index(-5, na + 5), slice(1, -1)
        for b in range(6):
            A = self.meanA[b].permute(2, 3, 0, 1)[..., None]
            Ai = torch.linalg.inv(self.meanA[b]).permute(2, 3, 0, 1)[..., None]
            u = [C[b][:1]]
            for c in (1, 5):
                x = C[b][c:c + 3]
                q = _matvec(Ai, x)
                corr = _matvec(_diff(A, 1), _diff(q, 1)) + _matvec(_diff(A, 2), _diff(q, 2))
                u += [_matvec(Ai, x - corr / 12), C[b][4:5]]
            u = torch.cat(u[:-1])[:, s, s]
            us = out[b]
            us[..., 5:-5] = u
            for q in range(5):
                rho, ur, p = _wind_inner(m.radial(m.index(q - 5, q - 4))["rhalf"])
                us[..., q] = 0
                us[0, ..., q], us[1, ..., q], us[4, ..., q] = rho, rho * ur, p / (GAMMA - 1) + 0.5 * rho * ur ** 2
                f = m.radial(m.index(nr - 1, nr))["rhalf"] / m.radial(m.index(nr + q, nr + q + 1))["rhalf"]
                us[:6, ..., nr + 5 + q], us[6:, ..., nr + 5 + q] = u[:6, ..., -1] * f ** 2, u[6:, ..., -1] * f
        return out

    def step(self, u, dt):
        na = self.na
        reg = {key: 0 for key in self.edges}

        def rhs(x, weight):
            W, out = self.prepare(x), []
            for b in range(6):
                k, fx = _order4_box(self.metrics, b, (0, 0, 0), W[b], self.case)
                out.append(k)
                for ax in (1, 2):
                    for s in (0, 1):
                        reg[b, ax, s] = reg[b, ax, s] + weight * fx[ax].select(3 - ax, -s)
            return torch.stack(out)

        new = _rk4(u, dt, rhs)
        for (b, ax, side), (nb, nax, nside, along) in self.edges.items():
            other = reg[nb, nax, nside][:, torch.as_tensor(along, device=u.device)]
            mean = 0.5 * (reg[b, ax, side] + (1.0 if nside != side else -1.0) * other)
            edge = new[b].select(3 - ax, na - 1 if side else 0)
            edge += (-na if side else na) * (mean - reg[b, ax, side])
        return new
