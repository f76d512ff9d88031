"""The work this framework is used for, as measurable cases.

A case is a dict of plain values.  `listed()` gives the fixed ones, `draw(rng)`
one more from the same ranges, `prepare` what a program holds before the call,
`run` one pass through the public entry points, `work` the bytes and
floating-point operations that pass cannot do without and `exact` the same
results from plain torch and numpy in 64 bits.

Kinds:
  march  a case marched from its cold start: INICON2, `steps` pseudo-time
         steps, then the state, the nodal fields and the step histories (and,
         with `every` > 0, the records of the device output ring)
  batch  several cavities of different sizes advanced together
  rre    an extrapolation cycle: steps, snapshots of consecutive iterates,
         the extrapolated state
  net    the warm-start network: Adam steps on a training set, then the
         prediction for the set's inputs and the trained parameters
What an FP32 handle computes is handed back in single precision (its fields
carry no more); a shared nodal array keeps the six fields together.
"""
import functools
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dg-bgk_b200"))
from dgbgk import cases as dc  # noqa: E402
from dgbgk.solver import Batch, Solver, setup_mesh, vspace  # noqa: E402
from dgbgk.warmstart import MLP  # noqa: E402

FIELDS = ("nd", "rho", "u", "v", "ps", "temp")


# ------------------------------------------------------------- the cases ----
def _cavity(n, nr, nt, mach, kn, prec, steps, **more):
    return dict(kind="march", mesh="cavity", nx=n, ny=n, nr=nr, nt=nt, mach=mach, kn=kn, prec=prec, steps=steps,
                immat=1, alpha=1.0, sides="", side=0.0, half=0.0, every=0, **more)


def _channel(nx, ny, nr, nt, mach, kn, prec, steps, half=5.0, side=1.0, sides="outflow", immat=1, alpha=1.0, every=0,
             **more):
    # [-5, 15] x [-half, half] around a square obstacle of this side
    return dict(kind="march", mesh="channel", nx=nx, ny=ny, nr=nr, nt=nt, mach=mach, kn=kn, prec=prec, steps=steps,
                immat=immat, alpha=alpha, sides=sides, side=side, half=half, every=every, **more)


def listed():
    return [
        # the smallest case of the test suite and the smoke run: a step's launches are the whole time
        _cavity(8, 8, 16, 0.3, 0.1, 64, 40, name="cavity8_fp64"),
        # the first benchmark workload, the 32 x 32 lid-driven cavity: 661 000 such steps to its steady state
        _cavity(32, 16, 32, 0.3, 0.1, 64, 200, name="cavity32_fp64"),
        _cavity(32, 16, 32, 0.3, 0.1, 32, 200, name="cavity32_fp32"),
        # one channel of the warm-start family (training-set generation in FP32, the finish in FP64)
        _channel(100, 100, 16, 32, 2.5, 0.07, 32, 100, half=10.0, sides="freestream", name="family100_fp32"),
        _channel(100, 100, 16, 32, 2.5, 0.07, 64, 60, half=10.0, sides="freestream", name="family100_fp64"),
        # the headline workload, Mach 2 past a square at 1.4e8 unknowns
        _channel(200, 100, 24, 48, 2.0, 0.05, 32, 100, name="channel200_fp32"),
        _channel(200, 100, 24, 48, 2.0, 0.05, 64, 60, name="channel200_fp64"),
        # odd sizes everywhere, diffuse side walls and the consistent mass matrix (IMMAT = 0)
        _channel(61, 37, 11, 37, 2.0, 0.05, 32, 100, sides="wall", immat=0, name="ragged_immat0_fp32"),
        # partial wall accommodation with periodic output, as the reference's own inputs have it (ALPHA 0.9)
        _channel(93, 47, 20, 20, 2.0, 0.05, 32, 60, sides="wall", alpha=0.9, every=20, name="alpha09_output_fp32"),
        # cavities of mixed sizes, velocity grids, Mach and Knudsen numbers advanced in one batch
        dict(kind="batch", ncases=6, pick=1, prec=32, steps=40, name="batch_cavities_fp32"),
        # one cycle of the extrapolated march (m = 8) that finishes in FP64
        dict(kind="rre", nx=50, ny=50, nr=16, nt=32, mach=2.5, kn=0.07, prec=64, steps=20, m=8, name="rre_cycle_fp64"),
        # the warm-start network at the study's size, trained and evaluated
        dict(kind="net", width=512, depth=4, n_out=32768, batch=128, iters=40, lr=1e-4, name="network_512x4"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    r = rng.random()
    if r < 0.12:
        return dict(kind="batch", ncases=rng.randint(2, 6), pick=rng.randint(2, 1 << 20), prec=rng.choice((32, 32, 64)),
                    steps=rng.randint(20, 40))
    if r < 0.22:
        return dict(kind="rre", nx=rng.randint(20, 50), ny=rng.randint(20, 50), nr=rng.randint(8, 16),
                    nt=rng.randint(16, 32), mach=round(rng.uniform(2.0, 3.0), 3), kn=round(rng.uniform(0.04, 0.12), 4),
                    prec=64, steps=rng.randint(10, 30), m=rng.randint(4, 8))
    if r < 0.36:
        return dict(kind="net", width=128 * rng.randint(1, 4), depth=rng.randint(2, 4), n_out=128 * _log_int(rng, 16, 256),
                    batch=128 * rng.randint(1, 2), iters=rng.randint(10, 40), lr=1e-4)
    prec = rng.choice((32, 32, 64))
    immat, alpha, every = rng.choice((1, 1, 1, 0)), rng.choice((1.0, 1.0, 1.0, 1.0, 0.9)), rng.choice((0, 0, 10))
    nr, nt = _log_int(rng, 8, 32), _log_int(rng, 16, 64)
    if alpha < 1.0:  # the reference's mirrored-velocity lookup needs a square grid
        nr = nt = _log_int(rng, 16, 26)
    if rng.random() < 0.4:
        n = _log_int(rng, 8, 96)
        c = _cavity(n, nr, nt, round(rng.uniform(0.1, 1.0), 3), round(10.0 ** rng.uniform(-2.0, 0.0), 4), prec, 0)
        c["immat"], c["alpha"], c["every"], elems = immat, alpha, every, 2 * n * n
    else:
        nx, ny = _log_int(rng, 20, 200), _log_int(rng, 20, 110)
        c = _channel(nx, ny, nr, nt, round(rng.uniform(2.0, 3.0), 3), round(rng.uniform(0.04, 0.12), 4), prec, 0,
                     half=rng.choice((5.0, 10.0)), side=round(rng.uniform(1.1, 1.4), 3),
                     sides=rng.choice(("outflow", "freestream", "wall")), immat=immat, alpha=alpha, every=every)
        elems = 2 * nx * ny
    # no more work than the largest listed case, and 20 to 200 steps of it
    dofs = 3 * elems * nr * nt
    most = 8.0e9 * 32 / prec
    while 20 * dofs > most:
        c["nx"] = c["nx"] * 4 // 5
        if c["mesh"] == "cavity":
            c["ny"] = c["nx"]
        else:
            c["ny"] = max(20, c["ny"] * 4 // 5)
        dofs = 3 * 2 * c["nx"] * c["ny"] * nr * nt
    c["steps"] = int(min(rng.randint(20, 200), max(20, most / dofs)))
    return c


# -------------------------------------------------------------- the inputs ----
@functools.lru_cache(maxsize=32)
def _mesh(kind, nx, ny, half, side, sides, lid):
    if kind == "cavity":
        return dc.cavity_mesh(nx, lid_speed=lid)
    return dc.channel_mesh(-5.0, 15.0, -half, half, nx, ny, side, sides=sides)


@functools.lru_cache(maxsize=8)
def _setup(*key):
    m = _mesh(*key)
    return setup_mesh(m.intma, m.coord, m.bsido)


def _physics(c):
    """Mesh key, physical parameters, velocity radius, inflow and start of a march-like case."""
    cavity = c.get("mesh", "channel") == "cavity"
    ph = dc.physical_params(c["mach"], c["kn"], length=1.0 if cavity else c.get("side", 1.0))
    if cavity:
        key = ("cavity", c["nx"], c["ny"], 0.0, 0.0, "", ph["speed"])
        rv, cinf, u0, perturb = 4.0, (0.0, 0.0, 0.0, 0.0), 0.0, 1e-3
    else:
        key = ("channel", c["nx"], c["ny"], c.get("half", 10.0), c.get("side", 1.0), c.get("sides", "freestream"), 0.0)
        rv, cinf, u0, perturb = 4.0 + ph["speed"], (1.0, ph["p_bar"], ph["speed"], 0.0), ph["speed"], 1e-3
    return key, ph, rv, cinf, u0, perturb


def _scale(key, seed, perturb):
    """The seeded density perturbation per DG node."""
    rng = np.random.Generator(np.random.PCG64(seed))
    return 1.0 + rng.uniform(-perturb, perturb, size=(_mesh(*key).nelem, 3))


def _solver(c):
    key, ph, rv, cinf, _, _ = _physics(c)
    m = _mesh(*key)
    eta, w = dc.gll(c["nr"])
    vc, sw = vspace(c["nr"], c["nt"], eta, w)
    return Solver(m.intma, m.coord, m.bsido, _setup(*key), vc, sw, c["nr"], c["nt"], rv, immat=c.get("immat", 1),
                  csafm=0.5, alpha=c.get("alpha", 1.0), rgas=1.0, molar_mass=ph["molar_mass"], diameter=ph["diameter"],
                  cinf=cinf, precision=c["prec"], wall_velocity=m.wall_velocity)


def _buffer(s, prec):
    """A pinned host buffer for the state, which a program that reads it back keeps."""
    t = torch.empty((s.E, s.V, 3), dtype=torch.float64 if prec == 64 else torch.float32,
                    pin_memory=torch.cuda.is_available())
    return t.numpy()


def _batch_cases(c, seed):
    """Cavities with the spread of the batched workload: mesh size, velocity grid, Mach and Kn all drawn."""
    r = random.Random(c["pick"])
    out = []
    for k in range(c["ncases"]):
        out.append((_cavity(r.choice((16, 24, 32, 40, 48, 56, 64)), r.randint(8, 24), r.randint(16, 64),
                            r.uniform(0.1, 1.0), 10.0 ** r.uniform(-2.0, 0.0), c["prec"], c["steps"]), 1000 * seed + k))
    return out


def _net_data(c, seed):
    """Case parameters in [-1, 1]^3 and standardised fields: smooth functions of them, a spread of frequencies."""
    rng = np.random.Generator(np.random.PCG64(seed))
    x = rng.uniform(-1.0, 1.0, (c["batch"], 3)).astype(np.float32)
    a = rng.normal(0.0, 1.0, (3, c["n_out"]))
    b = rng.uniform(-np.pi, np.pi, c["n_out"])
    t = (math.sqrt(2.0) * np.sin(x.astype(np.float64) @ a + b)).astype(np.float32)
    return x, t


def prepare(case, seed):
    c = case
    if c["kind"] == "net":
        x, t = _net_data(c, seed)
        net = MLP(3, c["width"], c["depth"], c["n_out"], c["batch"], seed=seed)
        net.set_data(x, t)
        return {"case": c, "net": net, "x": x, "seed": seed}
    if c["kind"] == "batch":
        members = []
        for k, s in _batch_cases(c, seed):
            key, ph, _, _, u0, p = _physics(k)
            sv = _solver(k)
            members.append((sv, (1.0, ph["p_bar"], u0, 0.0, _scale(key, s, p)), _buffer(sv, c["prec"])))
            sv.inicon2(*members[-1][1])
        return {"case": c, "members": members, "batch": Batch([m[0] for m in members])}
    key, ph, _, _, u0, p = _physics(c)
    s = _solver(c)
    if c.get("every", 0):
        s.set_output(c["every"], capacity=8)
    return {"case": c, "solver": s, "start": (1.0, ph["p_bar"], u0, 0.0, _scale(key, seed, p)),
            "out": _buffer(s, c["prec"])}


# ------------------------------------------------------------------- a pass ----
def _single(x, prec):
    return x.astype(np.float32) if prec == 32 else x


def run(state):
    c = state["case"]
    if c["kind"] == "net":
        loss = state["net"].train(c["iters"], lr=c["lr"], seed=state["seed"])
        y = state["net"].forward(state["x"])
        return {"loss": _single(loss, 32), "y": y, "params": state["net"].get_params()}
    prec = c["prec"]
    if c["kind"] == "batch":
        for s, start, _ in state["members"]:
            s.inicon2(*start)
        r = state["batch"].advance(c["steps"])
        return {"f": [s.get_state(out=o) for s, _, o in state["members"]], "steps": r["steps"],
                "l2": _single(r["res_l2_last"], prec)}
    s = state["solver"]
    s.inicon2(*state["start"])
    if c["kind"] == "rre":
        s.advance(c["steps"])
        s.snapshot(0)
        for k in range(c["m"] + 1):
            s.advance(1)
            s.snapshot(k + 1)
        g = s.extrapolate(c["m"] + 2)
        return {"f": s.get_state(out=state["out"]), "gamma_sum": float(g.sum())}
    r = s.advance(c["steps"])
    m = s.macros()
    out = {"f": s.get_state(out=state["out"]), "fields": _single(np.stack([m[k] for k in FIELDS]), prec),
           "linf": _single(r["res_linf"], prec), "l2": _single(r["res_l2"], prec), "dte": _single(r["dte"], prec)}
    if c["every"]:
        # the ring keeps the last records of the handle: those of this march
        recs = s.outputs()[-(c["steps"] // c["every"]):][-8:]
        out["records"] = [_single(np.stack([q[k] for k in FIELDS]), prec) for q in recs]
    return out


# ----------------------------------------------------------------- the work ----
def _size(c):
    if c["mesh"] == "cavity":
        elems = 2 * c["nx"] * c["ny"]
    else:
        elems = _mesh(*_physics(c)[0]).nelem
    return 3 * elems * c["nr"] * c["nt"]


def work(case):
    c = case
    if c["kind"] == "net":
        layers = [(3, c["width"])] + [(c["width"], c["width"])] * (c["depth"] - 1) + [(c["width"], c["n_out"])]
        n = sum(i * o + o for i, o in layers)
        gemm = 2.0 * c["batch"] * sum(i * o for i, o in layers)
        # an Adam step reads and writes the weights and both moments; the targets are read once a step
        return {"bytes": c["iters"] * (24.0 * n + 4.0 * c["batch"] * c["n_out"]) + 4.0 * n,
                "flops": c["iters"] * 3 * gemm + gemm}
    if c["kind"] == "batch":
        dofs = sum(_size(k) for k, _ in _batch_cases(c, 1))
        sf, steps, extra = c["prec"] // 8, c["steps"], 2
    elif c["kind"] == "rre":
        dofs = _size(dict(c, mesh="channel"))
        # the snapshots written, read for the Gram matrix and (but the last) for the combination
        sf, steps, extra = c["prec"] // 8, c["steps"] + c["m"] + 1, 3 * (c["m"] + 2) + 1
    else:
        dofs, sf, steps, extra = _size(c), c["prec"] // 8, c["steps"], 2
    # a step reads the state for the moments and again for the sweep (whose time step and equilibria
    # need every moment first) and writes it
    return {"bytes": (3.0 * steps + extra) * sf * dofs, "flops": 60.0 * steps * dofs}


# ------------------------------------------------- the same results, in 64 bits ----
PI = 3.1416  # the reference's constant


def _grid(c, rv, dev):
    """Velocities and quadrature weights: rv/2 (eta + 1) and pi zeta, zeta = -1 + 2 k / nt."""
    eta, w = np.polynomial.legendre.Legendre.basis(c["nr"] - 1).deriv().roots(), None
    eta = np.concatenate([[-1.0], np.sort(eta.real), [1.0]])
    pn = np.polynomial.legendre.Legendre.basis(c["nr"] - 1)
    for _ in range(4):  # the interior nodes to machine precision: Newton on P'
        d1, d2 = pn.deriv()(eta[1:-1]), pn.deriv(2)(eta[1:-1])
        eta[1:-1] -= d1 / d2
    w = 2.0 / ((c["nr"] - 1) * c["nr"] * pn(eta) ** 2)
    zeta = -1.0 + np.arange(1, c["nt"] + 1) * (2.0 / c["nt"])
    e, z, ww = np.repeat(eta, c["nt"]), np.tile(zeta, c["nr"]), np.repeat(w, c["nt"])
    r = 0.5 * rv * (e + 1.0)
    wjf = ww * (PI * rv * rv * 0.25 * (e + 1.0)) * (4.0 / ww.sum())
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    return up(r * np.cos(PI * z)), up(r * np.sin(PI * z)), up(wjf), zeta


def _connect(mesh):
    """Per element edge (node k to k + 1): the neighbour's element and its local nodes at both ends, or the
    boundary side."""
    t = mesh.intma.astype(np.int64) - 1
    E = t.shape[0]
    a, b = t, np.roll(t, -1, axis=1)
    big = int(t.max()) + 1
    here = {int(k): i for i, k in enumerate((a * big + b).reshape(-1))}
    nbr = np.full(3 * E, -1, dtype=np.int64)
    for i, k in enumerate((b * big + a).reshape(-1)):
        nbr[i] = here.get(int(k), -1)
    nbr = nbr.reshape(E, 3)
    # the neighbour's edge runs the other way: its node k + 1 is this edge's node k
    ne, nk = nbr // 3, nbr % 3
    src_p, src_q = 3 * ne + (nk + 1) % 3, 3 * ne + nk
    side = np.full((E, 3), -1, dtype=np.int64)
    for i, s in enumerate(mesh.bsido):
        e = int(s[2]) - 1
        k = int(np.flatnonzero(t[e] == int(s[0]) - 1)[0])
        side[e, k] = i
    return t, nbr >= 0, src_p, src_q, side


class _March:
    """The pseudo-time march in 64 bits: f as (elements, 3, velocities)."""

    def __init__(self, c, seed):
        self.c = c
        dev = self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        key, ph, rv, cinf, u0, p = _physics(c)
        mesh = self.mesh = _mesh(*key)
        self.cx, self.cy, self.w, self.zeta = _grid(c, rv, dev)
        self.alpha, self.immat, self.d = c.get("alpha", 1.0), c.get("immat", 1), ph["diameter"]
        up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
        t, inner, sp, sq, side = _connect(mesh)
        self.t = up(t)
        X = mesh.coord[t]
        E = t.shape[0]
        x21, x31, y21, y31 = (X[:, 1, 0] - X[:, 0, 0], X[:, 2, 0] - X[:, 0, 0], X[:, 1, 1] - X[:, 0, 1],
                              X[:, 2, 1] - X[:, 0, 1])
        rj = x21 * y31 - x31 * y21
        nxi, net = np.array([-1.0, 1.0, 0.0]), np.array([-1.0, 0.0, 1.0])
        gx = ((y31 / rj)[:, None] * nxi + (-y21 / rj)[:, None] * net)
        gy = ((-x31 / rj)[:, None] * nxi + (x21 / rj)[:, None] * net)
        self.rj, self.gx, self.gy = up(rj), up(gx), up(gy)
        self.dtc = float((0.5 * (1.0 / np.sqrt(gx ** 2 + gy ** 2)).min(axis=1) / rv).min())
        D = np.roll(X, -1, axis=1) - X
        # (length / 6) times the outward normal of each edge
        self.an = up(D[:, :, 1] / 6.0), up(-D[:, :, 0] / 6.0)
        kind = np.where(inner, 0, np.where(side >= 0, mesh.bsido[np.maximum(side, 0), 3], 0))  # 1 in, 2 out, 4 wall
        self.flux = up(((kind == 0) | (kind == 2)).astype(np.float64))
        self.inner = up(inner)
        self.src = up(np.where(inner, sp, 0)), up(np.where(inner, sq, 0))
        inflow = np.zeros(mesh.npoin, dtype=bool)
        inflow[(mesh.bsido[mesh.bsido[:, 3] == 1][:, :2] - 1).reshape(-1)] = True
        self.inflow = up(inflow[t])
        self.we, self.wk = (up(a) for a in np.nonzero(kind == 4))  # wall edges
        ws = side[kind == 4]
        tw = mesh.bsido[ws, 4].astype(np.float64)
        uw = mesh.wall_velocity[ws] if mesh.wall_velocity is not None else np.zeros((len(ws), 2))
        L = np.sqrt((D ** 2).sum(axis=2))[kind == 4]
        n = np.stack([D[kind == 4][:, 1], -D[kind == 4][:, 0]], axis=1) / L[:, None]
        self.wtw, self.wuw, self.wn, self.wl = up(tw), up(uw), up(n), up(L / 6.0)
        b2 = 0.5 / 1.0  # rho / (2 P) at T = 1
        self.nfinf = (1.0 / PI) * b2 * torch.exp(-b2 * ((self.cx - cinf[2]) ** 2 + self.cy ** 2))
        start = (1.0 / PI) * b2 * torch.exp(-b2 * ((self.cx - u0) ** 2 + self.cy ** 2))
        self.f = up(_scale(key, seed, p))[:, :, None] * start
        self.linf, self.l2, self.dte = [], [], []
        if self.alpha < 1.0 and len(ws):
            self._mirror()

    def _mirror(self):
        """The two grid velocities around each mirrored one and their weights, per wall edge."""
        n, cx, cy = self.wn.cpu().numpy(), self.cx.cpu().numpy(), self.cy.cpu().numpy()
        nt = self.c["nt"]
        ring = np.arange(len(cx)) // nt
        self.mi, self.mz, self.mt = [], [], []
        for ax, ay in n:
            test = cx * ax + cy * ay
            rx, ry = cx + np.abs(2 * test) * ax, cy + np.abs(2 * test) * ay
            rt = np.sqrt(rx * rx + ry * ry)
            with np.errstate(divide="ignore", invalid="ignore"):
                th = np.abs(np.arccos(np.minimum(np.abs(rx / rt), 1.0)))
            th = np.where(rx < 0, PI - th, th)
            th = np.where(ry < 0, -th, th) / PI
            j = np.searchsorted(self.zeta, th, side="left") - 1  # zeta[j] < th <= zeta[j + 1]
            j = np.where((j < 0) & (th == self.zeta[0]), 0, j)
            last = j >= nt - 1
            wrap = (j < 0) | last
            jj = np.clip(j, 0, nt - 2)
            i1 = np.where(wrap, ring * nt + nt - 1, ring * nt + jj)
            i2 = np.where(wrap, ring * nt, ring * nt + jj + 1)
            z1 = np.where(wrap, self.zeta[0] + 1.0, self.zeta[jj + 1] - self.zeta[jj])
            z2 = np.where(wrap, th + 1.0, th - self.zeta[jj])
            self.mi.append((i1, i2))
            self.mz.append((z1, z2))
            self.mt.append(test < 0)
        self.mi, self.mz, self.mt = np.array(self.mi), np.array(self.mz), np.array(self.mt)

    def moments(self):
        f, cx, cy = self.f, self.cx, self.cy
        self.n = f @ self.w
        inv = 1.0 / self.n
        self.ux, self.uy = (f @ (self.w * cx)) * inv, (f @ (self.w * cy)) * inv
        self.p, ct = torch.empty_like(self.n), torch.empty_like(self.n)
        for i in range(3):
            d2 = (cx - self.ux[:, i, None]) ** 2 + (cy - self.uy[:, i, None]) ** 2
            wf = self.w * f[:, i]
            self.p[:, i] = (0.5 * d2 * wf).sum(dim=1)
            ct[:, i] = (d2.sqrt() * wf).sum(dim=1)
        self.mu = math.sqrt(2.0) * PI * self.d * self.d * ct

    def step(self):
        self.moments()
        f, cx, cy = self.f, self.cx, self.cy
        dt = min(0.9 / float(self.mu.max()), self.dtc)
        b2 = self.n / (2.0 * self.p)
        q = torch.empty_like(f)
        for i in range(3):
            d2 = (cx - self.ux[:, i, None]) ** 2 + (cy - self.uy[:, i, None]) ** 2
            q[:, i] = (self.n[:, i] * b2[:, i] / PI)[:, None] * torch.exp(-b2[:, i, None] * d2)
        col = self.mu[:, :, None] * (q - f)
        del q
        div = sum((self.gx[:, i, None] * cx + self.gy[:, i, None] * cy) * f[:, i] for i in range(3))
        g = f - (0.5 * dt * (div - col.sum(dim=1) / 3.0))[:, None, :]
        rows = g.reshape(-1, g.shape[2])
        s3 = (0.5 / 3.0) * self.rj[:, None] * g.sum(dim=1)
        rhs = torch.stack([(self.gx[:, i, None] * cx + self.gy[:, i, None] * cy) * s3 for i in range(3)], dim=1)
        for k in range(3):
            a = (self.an[0][:, k, None] * cx + self.an[1][:, k, None] * cy) * self.flux[:, k, None]
            own = (a > 0) | ~self.inner[:, k, None]
            up = torch.where(own, g[:, k], rows[self.src[0][:, k]])
            uq = torch.where(own, g[:, (k + 1) % 3], rows[self.src[1][:, k]])
            rhs[:, k] -= a * (2 * up + uq)
            rhs[:, (k + 1) % 3] -= a * (up + 2 * uq)
        if len(self.we):
            e, k = self.we, self.wk
            k1 = (k + 1) % 3
            test = self.wn[:, :1] * cx + self.wn[:, 1:] * cy
            out = torch.where(test > 0, test, torch.zeros_like(test))
            eta = (out * 0.5 * (f[e, k] + f[e, k1])) @ self.w / torch.sqrt(2 * PI * self.wtw ** 3)
            mw = torch.exp(-((cx - self.wuw[:, :1]) ** 2 + (cy - self.wuw[:, 1:]) ** 2) / (2.0 * self.wtw[:, None]))
            wall = self.alpha * mw * eta[:, None]
            up, uq = torch.where(test >= 0, g[e, k], wall), torch.where(test >= 0, g[e, k1], wall)
            a = self.wl[:, None] * test
            flat = rhs.view(-1, rhs.shape[2])
            flat.index_add_(0, 3 * e + k, -a * (2 * up + uq))
            flat.index_add_(0, 3 * e + k1, -a * (up + 2 * uq))
        col *= dt
        rhs *= dt
        if self.alpha < 1.0 and len(self.we):
            self._specular(rhs, col, dt)
        self._finish(rhs, col, dt)

    def _specular(self, x, cdt, dt):
        """The mirrored part of the wall flux, (1 - ALPHA) (z2 f(I1) + z1 f(I2)) / (z1 + z2), in the reference's
        order: velocity after velocity, a lower one's new value and a higher one's old one."""
        e, k = self.we.cpu().numpy(), self.wk.cpu().numpy()
        elems, at = np.unique(e, return_inverse=True)
        te = torch.from_numpy(elems).to(self.dev)
        old = self.f[te].cpu().numpy()
        xs, cs = x[te].cpu().numpy(), cdt[te].cpu().numpy()
        mm = (6.0 / self.rj[te]).cpu().numpy()[:, None]
        infl = self.inflow[te].cpu().numpy()
        nf = self.nfinf.cpu().numpy()
        test = (self.wn[:, :1] * self.cx + self.wn[:, 1:] * self.cy).cpu().numpy()
        a = self.wl.cpu().numpy()[:, None] * test
        new = np.where(infl[:, :, None], nf, np.maximum(old + (mm[:, :, None] * xs + cs), 0.0))
        k1 = (k + 1) % 3
        om = 1.0 - self.alpha
        for v in range(old.shape[2]):
            w = np.flatnonzero(self.mt[:, v])
            if not len(w):
                continue
            z1, z2 = self.mz[w, 0, v], self.mz[w, 1, v]
            i1, i2 = self.mi[w, 0, v], self.mi[w, 1, v]
            A, K, K1 = at[w], k[w], k1[w]

            def F(node, i):
                return np.where(i < v, new[A, node, i], old[A, node, i])

            rp = om * (z2 * F(K, i1) + z1 * F(K, i2)) / (z1 + z2)
            rq = om * (z2 * F(K1, i1) + z1 * F(K1, i2)) / (z1 + z2)
            np.add.at(xs, (A, K, v), -dt * a[w, v] * (2 * rp + rq))
            np.add.at(xs, (A, K1, v), -dt * a[w, v] * (rp + 2 * rq))
            T = np.unique(A)
            u = np.maximum(old[T, :, v] + (mm[T] * xs[T, :, v] + cs[T, :, v]), 0.0)
            new[T, :, v] = np.where(infl[T], nf[v], u)
        x[te] = torch.from_numpy(xs).to(self.dev)

    def _finish(self, x, cdt, dt):
        f = self.f
        mm = (6.0 / self.rj)[:, None, None]
        d = mm * x + cdt
        if self.immat == 1:
            linf = d.abs().max()
        else:
            rows = torch.where(x >= 0, 3.0 * mm, -mm) * x + cdt
            linf = rows.max().clamp(min=0.0)
            del rows
        new = f + d
        d = torch.where(new < 0, -f, d)
        d[self.inflow] = 0.0
        self.l2.append(float(d.square().sum().sqrt()))
        self.linf.append(float(linf))
        self.dte.append(dt)
        new.clamp_(min=0.0)
        new[self.inflow] = self.nfinf
        self.f = new

    def march(self, n):
        for _ in range(n):
            self.step()

    def state(self):
        return self.f.transpose(1, 2).contiguous().cpu()

    def fields(self):
        self.moments()
        idx, w = self.t.reshape(-1), self.rj[:, None].expand(-1, 3).reshape(-1)
        acc = lambda q: torch.zeros(self.mesh.npoin, dtype=torch.float64, device=self.dev).index_add_(  # noqa: E731
            0, idx, w * q.reshape(-1))
        area = acc(torch.ones_like(self.n))
        n, u, v, p = (acc(q) / area for q in (self.n, self.ux, self.uy, self.p))
        return torch.stack([n, n, u, v, p, p / n]).cpu().numpy()


def _exact_net(c, seed):
    """Forward, gradients and Adam in 64 bits from the network's initial parameters, every step on the whole set
    (a training set of one minibatch: the order of its rows does not matter)."""
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    x, t = (torch.from_numpy(a).double().to(dev) for a in _net_data(c, seed))
    dims = [(64, c["width"])] + [(c["width"], c["width"])] * (c["depth"] - 1) + [(c["width"], c["n_out"])]
    net = MLP(3, c["width"], c["depth"], c["n_out"], c["batch"], seed=seed)  # its seeded initial parameters: an input
    p = torch.from_numpy(net.get_params()).double().to(dev)
    net.close()
    m, v, loss = torch.zeros_like(p), torch.zeros_like(p), []

    def forward(p):
        h, at = torch.nn.functional.pad(x, (0, 61)), 0
        for l, (i, o) in enumerate(dims):
            h = h @ p[at:at + i * o].view(o, i).T + p[at + i * o:at + i * o + o]
            at += i * o + o
            h = torch.tanh(h) if l < len(dims) - 1 else h
        return h

    for k in range(1, c["iters"] + 1):
        p.requires_grad_(True)
        e = (forward(p) - t).square().mean()
        g, = torch.autograd.grad(e, p)
        p = p.detach()
        m = 0.9 * m + 0.1 * g
        v = 0.999 * v + 0.001 * g * g
        p = p - c["lr"] * (m / (1 - 0.9 ** k)) / ((v / (1 - 0.999 ** k)).sqrt() + 1e-8)
        loss.append(float(e.detach()))
    return {"loss": np.array(loss), "y": forward(p).cpu().numpy(), "params": p.cpu().numpy()}


def exact(case, seed):
    c = case
    if c["kind"] == "net":
        return _exact_net(c, seed)
    if c["kind"] == "batch":
        ms = []
        for k, s in _batch_cases(c, seed):
            m = _March(k, s)
            m.march(c["steps"])
            ms.append((m.state(), m.l2[-1]))
            del m
        return {"f": [a for a, _ in ms], "steps": None, "l2": np.array([b for _, b in ms])}
    if c["kind"] == "rre":
        m = _March(c, seed)
        m.march(c["steps"])
        snaps = [m.f]
        for _ in range(c["m"] + 1):
            m.march(1)
            snaps.append(m.f)
        u = torch.stack([(b - a).reshape(-1) for a, b in zip(snaps, snaps[1:])])
        G = (u @ u.T).cpu().numpy()
        G += 1e-14 * np.trace(G) * np.eye(len(G))  # the entry point's ridge
        g = np.linalg.solve(G, np.ones(len(G)))
        g /= g.sum()
        m.f = sum(float(a) * s for a, s in zip(g, snaps)).clamp(min=0.0)
        return {"f": m.state(), "gamma_sum": 1.0}
    m = _March(c, seed)
    recs = []
    for k in range(c["steps"]):
        m.march(1)
        if c["every"] and (k + 1) % c["every"] == 0:
            recs.append(m.fields())
    out = {"f": m.state(), "fields": m.fields(), "linf": np.array(m.linf), "l2": np.array(m.l2), "dte": np.array(m.dte)}
    if c["every"]:
        out["records"] = recs[-8:]
    return out
