"""The work that a user of this framework has it do, as cases to be timed.

A case is one phase of a simulation program: a domain (or a batch of them)
that is already under way takes a number of timesteps, the program reads the
solid fraction as the time loop does, closes the solute balance and reads the
fields that its output writes; or a recorded run is differentiated.  Each case
goes through the package's public calls only, from an input deck to host
arrays.

kind "seed"         one grain in an undercooled melt that cools on
kind "directional"  surface and bulk grains in a moving temperature gradient
kind "melt"         a laser track over a columnar substrate
kind "ensemble"     independent domains stepped as one batch
kind "adjoint"      gradient and replayed loss of a recorded run

Sites and orientations are drawn here from the seed and handed over, so that
another program can follow the same run: `exact` does, in 64 bits.
"""
from __future__ import annotations

import math
import os
import tempfile

import numpy as np
import torch

import mumatscale_b200 as M
from mumatscale_b200 import workloads as W

SEED_DX, DIR_DX, MELT_DX = 1e-6, 2e-6, 1e-6
FORMS = {"f64": M.PREC_F64, "f32": M.PREC_F32}
PARAMS = ("Dliq", "part_coef", "gibbs")


# ------------------------------------------------------------------ the cases
def _domain(name, kind, dims, form, warm, steps, read, fields="ce,fs,gr", split=(1, 1, 1), tuned=False, curv=0):
    case = {"kind": kind, "nx": dims[0], "ny": dims[1], "nz": dims[2], "form": form, "warm": warm, "steps": steps,
            "read": read, "fields": fields, "sx": split[0], "sy": split[1], "sz": split[2], "tuned": tuned,
            "curv": curv}
    return dict(case, name=name) if name else case


def _ensemble(name, domains, edge_max, form, warm, steps):
    case = {"kind": "ensemble", "domains": domains, "edge_max": edge_max, "form": form, "warm": warm, "steps": steps}
    return dict(case, name=name) if name else case


def _adjoint(name, dims, form, warm, steps, every, curv):
    case = {"kind": "adjoint", "nx": dims[0], "ny": dims[1], "nz": dims[2], "form": form, "warm": warm,
            "steps": steps, "every": every, "curv": curv}
    return dict(case, name=name) if name else case


def listed():
    return [
        # a small study or a test, its solid fraction read after every step:
        # the shortest calls, odd in every size
        _domain("seed 37x31x29 f64 read each step", "seed", (37, 31, 29), "f64", 200, 16, 1),
        # the one-grain deck with curvature, a result every 200 steps
        _domain("seed 64^3 f64 curvature", "seed", (64, 64, 64), "f64", 400, 200, 200, curv=1),
        # the directional deck at its own size, both forms, tile tuned first
        _domain("directional 256^3 f64", "directional", (256, 256, 256), "f64", 200, 100, 50, tuned=True),
        _domain("directional 256^3 f32", "directional", (256, 256, 256), "f32", 200, 100, 50, tuned=True),
        # a domain whose sizes fit no tile, the default tile
        _domain("directional 203x171x149 f32", "directional", (203, 171, 149), "f32", 200, 100, 50),
        # the laser track at its own size, split into subblocks as the
        # comparison with the reference runs it
        _domain("melt 512x256x128 f32", "melt", (512, 256, 128), "f32", 200, 100, 50, split=(2, 2, 4), tuned=True),
        # the same model, smaller and uneven, with the temperature written too
        _domain("melt 251x127x67 f64", "melt", (251, 127, 67), "f64", 120, 60, 30, fields="ce,fs,gr,temperature"),
        _domain("melt 317x149x83 f32", "melt", (317, 149, 83), "f32", 120, 60, 30, fields="ce,fs,gr,temperature"),
        # an ensemble study: the full one, and a few domains in the plain form
        _ensemble("ensemble of 64 f32", 64, 128, "f32", 400, 100),
        _ensemble("ensemble of 6 f64", 6, 96, "f64", 400, 100),
        # parameter calibration: backward through a recorded run, then the
        # loss at a trial step
        _adjoint("adjoint 128^3 f64 curvature", (128, 128, 128), "f64", 200, 200, 50, 1),
        _adjoint("adjoint 57x63x49 f32", (57, 63, 49), "f32", 100, 60, 25, 0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["seed", "directional", "directional", "melt", "melt", "ensemble", "adjoint"])
    form = rng.choice(["f64", "f32"])
    if kind == "ensemble":
        return _ensemble(None, _log_int(rng, 3, 40), rng.choice([64, 96, 128]), form, rng.randrange(300, 500),
                         rng.randrange(40, 100))
    if kind == "adjoint":
        dims = tuple(_log_int(rng, 24, 110) for _ in range(3))
        return _adjoint(None, dims, form, rng.randrange(50, 200), rng.randrange(40, 160), rng.randrange(15, 60),
                        rng.choice([0, 1]))
    cells = math.exp(rng.uniform(math.log(2.4e4), math.log(2e6 if kind == "melt" and form == "f64" else 1e7)))
    edge = cells ** (1 / 3)
    nx = max(24, int(edge * math.exp(rng.uniform(-0.2, 0.6))))
    ny = max(24, int(edge * math.exp(rng.uniform(-0.3, 0.2))))
    nz = max(24, int(cells / nx / ny))
    split = rng.choice([(1, 1, 1), (1, 1, 1), (1, 1, 1), (2, 1, 1), (2, 2, 1), (2, 2, 2)])
    dims = tuple(n // s * s for n, s in zip((nx, ny, nz), split))
    curv = rng.choice([0, 1]) if kind == "seed" else 0
    steps = max(16, min(200, int(6e8 / (dims[0] * dims[1] * dims[2]))))
    read = 1 if steps <= 20 else rng.choice([steps, (steps + 1) // 2])
    fields = rng.choice(["ce,fs,gr", "ce,fs,gr", "temperature,ce,fs,gr"])
    return _domain(None, kind, dims, form, rng.randrange(100, 160) if kind == "melt" else rng.randrange(100, 300), steps,
                   read, fields, split, rng.random() < 0.3, curv)


# -------------------------------------------------------------------- inputs
def _deck(dims, split, dx, seed, *, curv=0, t0=W.T_LIQ, gradient=0.0, velocity=0.0, cooling=0.0, bulk=0.0, surface=0.0,
          undercooling=(2.0, 0.5), fourier=W.FOURIER, max_grains=100000, extra=""):
    sb = [n // s for n, s in zip(dims, split)]
    assert all(b * s == n for b, s, n in zip(sb, split, dims))
    return f"""BaseFileName case
NSubblocks {split[0]} {split[1]} {split[2]}
NCellsPerSB {sb[0]} {sb[1]} {sb[2]}
FaceCtrl 1 1 1 1 1 1
CellSize {dx!r}
FSGrow 0.66
TimeStep {fourier * dx * dx / W.D_LIQ!r}
RandSeedVal {seed % 1000003 + 1}
TipCurvature {curv}
GibbsThomsonCoef {W.GIBBS!r}
FinishTime 0
FsFinish 1.1
LiquidusTemp {W.T_LIQ!r}
SolidusTemp {W.T_SOL!r}
Cinit {W.C0!r}
m_solute0 0 0 {W.SLOPE!r}
part_coef0 0 0 {W.K_PART!r}
Dsol {W.D_SOL!r}
Dliq {W.D_LIQ!r}
InitialTemperature {t0!r}
Gradient {gradient!r}
Velocity {velocity!r}
CoolingRate {cooling!r}
ScreenPFreq 0
MaxGrainDensity {bulk!r}
GNGaussCentre {undercooling[0]!r}
GNGaussSigma {undercooling[1]!r}
MaxGrainDensitySurf {surface!r}
GNGaussCentreSurf {undercooling[0]!r}
GNGaussSigmaSurf {undercooling[1]!r}
MaxTotGrains {max_grains}
GNOriented 1
{extra}"""


def _read_deck(text):
    fd, path = tempfile.mkstemp(suffix=".in")
    try:
        with os.fdopen(fd, "w") as f:
            f.write(text)
        p = M.read_deck(path)
        p.site_setup = 1  # the deck's own sites, which ours replace, need no parity
        return p
    finally:
        os.unlink(path)


def _sites(rng, dims, mu, sigma, bulk, surface=0):
    """`bulk` sites anywhere and `surface` sites in the lowest plane, no cell
    twice, with undercoolings N(mu, sigma) and random orientations."""
    nx, ny, nz = dims
    key = rng.integers(0, nx * ny * nz, bulk)
    key = np.unique(np.concatenate([key, rng.integers(0, nx * ny, surface)]))
    cells = np.stack([key % nx, key // nx % ny, key // (nx * ny)], 1).astype(np.int32)
    thr = np.maximum(0.05, rng.normal(mu, sigma, len(key))).astype(np.float32)
    rot = np.stack([W.quat_to_rotmat(q).ravel() for q in W.random_quaternions(rng, len(key))])
    return cells, thr, rot


def _inputs(case, seed):
    """One domain's deck, sites and substrate: everything a run depends on."""
    rng = np.random.default_rng([seed, 77])
    dims, kind = (case["nx"], case["ny"], case["nz"]), case["kind"]
    split = (case.get("sx", 1), case.get("sy", 1), case.get("sz", 1))
    n = dims[0] * dims[1] * dims[2]
    d = {"dims": dims, "split": split, "cols": None, "dx": SEED_DX}
    if kind in ("seed", "adjoint"):
        d["deck"] = _deck(dims, split, SEED_DX, seed, curv=case["curv"], t0=W.T_LIQ - 4.0, cooling=50.0,
                          max_grains=1000)
        c = [int(x // 2 + rng.integers(-2, 3)) for x in dims]
        # its threshold is met on the first step
        d["sites"] = (np.array([c], dtype=np.int32), np.zeros(1, dtype=np.float32),
                      W.quat_to_rotmat(W.random_quaternions(rng, 1)[0]).reshape(1, 9))
    elif kind == "directional":
        # G = 1e4 K/m, V = 1e-3 m/s, sites 1e13 m^-3 and 1e10 m^-2, N(2 K, 0.5 K)
        d["dx"] = DIR_DX
        d["deck"] = _deck(dims, split, DIR_DX, seed, t0=W.T_LIQ - 2.5, gradient=1e4, velocity=1e-3, bulk=1e13,
                          surface=1e10)
        d["sites"] = _sites(rng, dims, 2.0, 0.5, max(1, round(1e13 * n * DIR_DX ** 3)),
                            max(1, round(1e10 * dims[0] * dims[1] * DIR_DX ** 2)))
    elif kind == "melt":
        # the single-track deck's laser, scanned over neighbouring tracks with
        # a power in proportion to the domain's width; a quarter of its time
        # step, with which ce stays positive over thousands of steps
        nx, ny, nz = dims
        top = nz - max(3, nz // 16)
        extra = f"""AnalyticalThermal 1
LaserPower {150.0 * min(1.0, ny / 256)!r}
LaserSpeed 0.5
LaserSpotSize 50e-6
LaserAbsorption 0.4
LaserHatchSpacing {20e-6 * ny / 256!r}
LaserStartLocation {-50e-6!r} {0.2 * ny * MELT_DX!r} {top * MELT_DX!r}
NoOfLayers 1
NoOfTracks 12
SubInitialTemp 300
ThermalConductivity 100
SpecificHeat 395
Density {100 / 3e-5 / 395!r}
"""
        d["deck"] = _deck(dims, split, MELT_DX, seed, t0=300.0, bulk=1e14, undercooling=(3.0, 1.0), fourier=0.01,
                          extra=extra)
        d["sites"] = _sites(rng, dims, 3.0, 1.0, max(1, round(1e14 * n * MELT_DX ** 3)))
        cols, rot = W.columnar_columns(nx, ny, MELT_DX, 20e-6, int(rng.integers(1, 1 << 30)))
        gr = np.zeros((nz + 2, ny + 2, nx + 2), dtype=np.int32)
        gr[1:top + 1, 1:-1, 1:-1] = cols[None]
        d["cols"] = (gr, (gr > 0).astype(np.float64), rot)
    else:
        raise ValueError(kind)
    return d


def _members(case, seed):
    """The domains of an ensemble: edges drawn per axis, cooling rate
    log-uniform in 10-1000 K/s, site density log-uniform in 1e11-1e14 m^-3."""
    rng = np.random.default_rng([case["domains"], case["edge_max"], 5])  # the sizes are the case's
    edges = [e for e in (32, 48, 64, 96, 128) if e <= case["edge_max"]]
    sizes = [tuple(int(rng.choice(edges)) for _ in range(3)) for _ in range(case["domains"])]
    rng = np.random.default_rng([seed, 78])
    out = []
    for dims in sizes:
        rate, rho = float(10 ** rng.uniform(1, 3)), float(10 ** rng.uniform(11, 14))
        n = dims[0] * dims[1] * dims[2]
        out.append({"dims": dims, "split": (1, 1, 1), "cols": None, "dx": SEED_DX,
                    "deck": _deck(dims, (1, 1, 1), SEED_DX, seed + len(out), cooling=rate, bulk=rho,
                                  max_grains=20000),
                    "sites": _sites(rng, dims, 2.0, 0.5, max(1, round(rho * n * SEED_DX ** 3)))})
    return out


def _fill(dom, d):
    dom.set_sites(d["sites"][0], d["sites"][1])
    dom.set_site_orientations(d["sites"][0], d["sites"][2])
    if d["cols"] is not None:
        dom.set_grains(d["cols"][2])
        dom.upload("gr", d["cols"][0])
        dom.upload("fs", d["cols"][1])


def _host(n, field):
    """A pinned host buffer for n values of a field."""
    t = torch.empty(n, dtype=torch.int32 if field == "gr" else torch.float64, pin_memory=torch.cuda.is_available())
    return t.numpy()


def prepare(case, seed):
    if case["kind"] == "ensemble":
        members = _members(case, seed)
        batch = M.Batch([_read_deck(d["deck"]) for d in members], precision=FORMS[case["form"]])
        for dom, d in zip(batch.domains, members):
            _fill(dom, d)
        batch.autotune()
        batch.step(case["warm"])
        n = [dom.num_cells() for dom in batch.domains]
        at = np.concatenate([[0], np.cumsum(n)])
        bufs = {f: _host(int(at[-1]), f) for f in ("ce", "gr")}
        return {"case": case, "batch": batch, "bufs": bufs, "fs": np.zeros(len(n)),
                "part": {f: [b[at[i]:at[i + 1]] for i in range(len(n))] for f, b in bufs.items()}}
    d = _inputs(case, seed)
    p = _read_deck(d["deck"])
    if case["kind"] == "adjoint":
        q = _read_deck(d["deck"])
        q.Dliq *= 1.2
        q.part_coef *= 0.9
        with M.Domain(q, precision=FORMS[case["form"]]) as other:
            _fill(other, d)
            other.step(case["warm"] + case["steps"])
            target = other.download("ce")
    dom = M.Domain(p, precision=FORMS[case["form"]])
    _fill(dom, d)
    if case["kind"] == "adjoint":
        dom.step(case["warm"])
        dom.adjoint_record(case["steps"], case["every"])
        return {"case": case, "dom": dom, "target": target}
    if case["tuned"]:
        dom.autotune()
    dom.step(case["warm"])
    return {"case": case, "dom": dom, "bufs": {f: _host(dom.num_cells(), f) for f in case["fields"].split(",")}}


# ------------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    if case["kind"] == "ensemble":
        batch, part = state["batch"], state["part"]
        batch.step(case["steps"])
        for i, dom in enumerate(batch.domains):
            state["fs"][i] = dom.reduce("fs_fraction")
            for f, views in part.items():
                dom.download(f, out=views[i])
        return {"fs_fraction": state["fs"], **state["bufs"]}
    dom = state["dom"]
    if case["kind"] == "adjoint":
        g = dom.adjoint_gradient(state["target"])
        trial = dom.adjoint_replay_loss(state["target"], (1.02, 0.99, 1.0))
        return {"loss": g["loss"], **{k: g[k] for k in PARAMS}, "trial": trial}
    fractions, left = [], case["steps"]
    while left > 0:
        n = min(case["read"], left)
        fractions.append(dom.step_reduce(n))
        left -= n
    out = {"fs_fraction": np.array(fractions), "solute": dom.reduce("ce_sum")}
    for f, buf in state["bufs"].items():
        out[f] = dom.download(f, out=buf)
    return out


def work(case):
    """Per cell and step: the fields read and written once (ce, cl, fs and the
    grain ids; the temperature too where it is a field); per cell once: the
    fields read for the host.  The flops: the 7-point update, and the
    temperature's 400 products and sums per cell on the laser track."""
    word = 8 if case["form"] == "f64" else 4
    if case["kind"] == "ensemble":
        cells = sum(d["dims"][0] * d["dims"][1] * d["dims"][2] for d in _members(case, 0))
        return {"bytes": cells * (case["steps"] * (6 * word + 4) + 2 * (word + 4)),
                "flops": cells * case["steps"] * 60}
    cells = case["nx"] * case["ny"] * case["nz"]
    if case["kind"] == "adjoint":
        # replay twice (fields in and out, a byte for the branch), the
        # backward step once: the state and its adjoint in, the adjoint out
        replay = 6 * word + 1 + 8 * case["curv"]
        back = (3 + 3 + 3) * word + 1 + 8 * case["curv"]
        return {"bytes": cells * case["steps"] * (2 * replay + back), "flops": cells * case["steps"] * 220}
    melt = case["kind"] == "melt"
    names = case["fields"].split(",")
    once = sum(4 + 4 if f == "gr" else word + 8 for f in names)
    return {"bytes": cells * (case["steps"] * (6 * word + 4 + (2 * word if melt else 0)) + once),
            "flops": cells * case["steps"] * (60 + (800 if melt else 0))}


# ------------------------------------------------------- the same in 64 bits
class _Run:
    """The time loop on plain tensors in 64 bits, faces closed, no curvature:
    temperature, nucleation, activation, diffusion, fraction solid, capture."""

    def __init__(self, d, scale=(1.0, 1.0)):
        p = _read_deck(d["deck"])
        self.p, self.dev = p, "cuda" if torch.cuda.is_available() else "cpu"
        gx, gy, gz = d["dims"]
        self.shape, self.split = (gz, gy, gx), d["split"]
        f = dict(dtype=torch.float64, device=self.dev)
        self.f = f
        dtx = p.ts_delt / (p.cellSize * p.cellSize)
        dl, k = p.Dliq * scale[0], p.part_coef * scale[1]
        self.par = {"rs": p.Dsol * dtx, "rl": dl * dtx, "dxt": dl / p.cellSize / p.cellSize * p.ts_delt, "k": k}
        self.ce = torch.full(self.shape, p.Cinit, **f)
        self.cl = self.ce.clone()
        self.fs = torch.zeros(self.shape, **f)
        self.gr = torch.zeros(self.shape, dtype=torch.int64, device=self.dev)
        self.dc = torch.zeros(gz * gy * gx, 3, **f)
        self.rot = torch.zeros(int(p.maxTotalGrains) + 1, 9, **f)
        self.ts, self.grains = 0, 1
        # subblock of every cell and its place in it: list and id order
        K, J, I = torch.meshgrid(*(torch.arange(n, device=self.dev) for n in self.shape), indexing="ij")
        sb = [n // s for n, s in zip((gx, gy, gz), self.split)]
        rank = I // sb[0] + (J // sb[1] + K // sb[2] * self.split[1]) * self.split[0]
        self.sbcells = sb[0] * sb[1] * sb[2]
        self.order = (rank * self.sbcells + (K % sb[2] * sb[1] + J % sb[1]) * sb[0] + I % sb[0]).flatten()
        nr = self.split[0] * self.split[1] * self.split[2]
        self.nr = nr
        self.slots = torch.zeros(nr, self.sbcells + 102, 3, **f)
        self.slot_size = torch.zeros(nr, dtype=torch.int64, device=self.dev)
        c, thr, rot = d["sites"]
        c = torch.as_tensor(c, dtype=torch.int64, device=self.dev)
        flat = (c[:, 2] * gy + c[:, 1]) * gx + c[:, 0]
        by = torch.argsort(self.order[flat])
        self.site = flat[by]
        self.site_thr = torch.as_tensor(thr, device=self.dev).double()[by]
        self.site_rot = torch.as_tensor(rot, **f)[by]
        if d["cols"] is not None:
            gr, fs, rot = d["cols"]
            self.gr = torch.as_tensor(gr[1:-1, 1:-1, 1:-1], dtype=torch.int64, device=self.dev).contiguous()
            self.fs = torch.as_tensor(fs[1:-1, 1:-1, 1:-1], **f).contiguous()
            self.rot[1:len(rot) + 1] = torch.as_tensor(rot, **f)
            self.grains = len(rot) + 1

    def temperature(self, ts, halo=False):
        """At step ts, of a shape that broadcasts over the domain."""
        p, t = self.p, ts * self.p.ts_delt
        gz, gy, gx = self.shape
        if not p.am:
            if p.gradient == 0:
                return torch.full((1, 1, 1), p.initialTemperature - t * p.cool_rate, **self.f)
            lo, n = (0, gz + 2) if halo else (1, gz)
            axis = (torch.arange(lo, lo + n, **self.f) + 0.5) * p.cellSize - p.cellSize * 0.5
            return (p.initialTemperature + p.gradient * (axis - p.velocity * t)).reshape(-1, 1, 1)
        xlen = gx * p.cellSize + p.lsd
        tline = xlen / p.lv + 1.5e-4 / p.lv
        track = math.floor(t / tline) if p.amtracks > 1 else 0
        xnow, ynow, znow = p.x0 + (t - track * tline) * p.lv, p.y0 + track * p.lhs, p.z0
        alpha, spot = p.lthcon / (p.rho * p.lcp), p.lsd / (2.0 * 1.414)
        ldt = 20 * alpha / p.lv / p.lv / 400
        power = 0.0 if t < 1e-4 else p.lpow
        front = p.lab * power * alpha / (5.568328 * p.lthcon)
        lt = (0.5 + torch.arange(400, **self.f)) * ldt
        a = spot * spot + 4 * alpha * lt

        def line(n):
            lo, m = (0, n + 2) if halo else (1, n)
            return (torch.arange(lo, lo + m, **self.f) + 0.5) * p.cellSize

        X = torch.exp(-(line(gx)[None] - xnow + (p.lv * lt)[:, None]) ** 2 / a[:, None])
        Y = torch.exp(-(line(gy)[None] - ynow) ** 2 / a[:, None])
        z = line(gz)
        Z = ldt * torch.exp(-(z[None] - znow) ** 2 / (4 * alpha * lt)[:, None]) / (torch.sqrt(alpha * lt) * a)[:, None]
        rows = (Z[:, :, None] * Y[:, None, :]).reshape(400, -1)
        T = (p.liniT + front * (rows.T @ X)).reshape(len(z), -1, X.shape[1])
        return torch.where((z <= znow + p.cellSize).reshape(-1, 1, 1), T, torch.zeros((), **self.f))

    def update(self, ce, cl, fs, T, par, branch=None, gr=None):
        """Diffusion and the change of the fraction solid; which of the rules
        holds in a cell is decided here, or given by `branch`."""
        p = self.p
        nb = 0
        for axis in range(3):
            n = self.shape[axis]
            lo, hi = (fn.narrow(axis, 0, n - 1) for fn in (cl, fs)), (fn.narrow(axis, 1, n - 1) for fn in (cl, fs))
            (cl0, fs0), (cl1, fs1) = lo, hi
            av = 0.5 * (fs0 + fs1)
            flow = (par["rs"] * av + par["rl"] * (1 - av)) * (cl1 - cl0)
            pad = [0] * 6
            after, before = list(pad), list(pad)
            after[2 * (2 - axis) + 1] = 1
            before[2 * (2 - axis)] = 1
            nb = nb + torch.nn.functional.pad(flow, after) - torch.nn.functional.pad(flow, before)
        cen = ce + nb
        if bool((cen < 0).any()):
            raise ValueError("ce < 0")
        k, m = par["k"], p.m_solute0
        u = 1 - (1 - k) * fs
        dcl = (p.Cinit + (T - p.liquidusTemp) / m - cl) * par["dxt"] * 2 + nb / u
        grown = fs + (dcl * u - nb) / (1 - k) / cl
        if branch is None:
            off = (gr <= 0) | (T < 1.0) | (T > p.liquidusTemp)
            keep = ~off & (fs == 1) & (p.liquidusTemp - T + m * (cl - p.Cinit) >= 0)
            neg = ~off & ~keep & (grown < 0)
            branch = (off | neg, keep, ~off & ~keep & ~neg & (grown > 1))
        reset, keep, clamp = branch
        cln = torch.where(reset, cen, torch.where(keep, cen / k, cl + dcl))
        fsn = torch.where(reset, torch.zeros_like(fs), torch.where(keep, fs, torch.where(clamp, torch.ones_like(fs), grown)))
        return cen, cln, fsn, branch

    def step(self):
        p = self.p
        self.ts += 1
        T = self.temperature(self.ts)
        full = T.expand(self.shape)
        # nucleation and activation
        gr = self.gr.flatten()
        z, y, x = (self.site // (self.shape[1] * self.shape[2]), self.site // self.shape[2] % self.shape[1],
                   self.site % self.shape[2])
        Ts = full[z, y, x]
        hit = (gr[self.site] <= 0) & (p.liquidusTemp - Ts + p.m_solute0_c * (self.cl[z, y, x] - p.Cinit) > self.site_thr)
        if p.am and self.ts * p.ts_delt > 1e-4:
            hit &= Ts >= p.solidusTemp
        new = torch.nonzero(hit).flatten()
        ids = self.grains + torch.arange(len(new), device=self.dev)
        gr[self.site[new]] = ids
        self.rot[ids] = self.site_rot[new]
        self.grains += len(new)
        # solute and fraction solid
        old = (self.ce, self.cl, self.fs)
        self.ce, self.cl, self.fs, branch = self.update(*old, T, self.par, gr=gr.reshape(self.shape))
        gr[branch[0].flatten()] = 0
        self.gr = gr.reshape(self.shape)
        self._capture()
        return old, T, branch

    def _capture(self):
        p, (gz, gy, gx) = self.p, self.shape
        s = torch.nn.functional.pad(self.gr > 0, [1] * 6)
        c = slice(1, -1)
        near = s[c, c, 2:] | s[c, c, :-2] | s[c, 2:, c] | s[c, :-2, c] | s[2:, c, c] | s[:-2, c, c]
        cells = torch.nonzero((near & ~s[c, c, c]).flatten()).flatten()
        if not len(cells):
            return
        cells = cells[torch.argsort(self.order[cells])]
        rank = self.order[cells] // self.sbcells
        count = torch.bincount(rank, minlength=self.nr)
        start = torch.cumsum(count, 0) - count
        slot = torch.arange(len(cells), device=self.dev) - start[rank] + 1
        grown = count > self.slot_size
        zero_to = torch.where(grown, self.slot_size, torch.zeros_like(count))
        self.slot_size = torch.where(grown, count + 100, self.slot_size)
        pos = (cells % gx, cells // gx % gy, cells // (gx * gy))
        pre = self.gr.flatten()
        taken = torch.zeros_like(cells)
        centre = torch.zeros(len(cells), 3, **self.f)
        for nx, ny, nz in ((1, 0, 0), (0, 1, 0), (-1, 0, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1)):
            X, Y, Z = pos[0] + nx, pos[1] + ny, pos[2] + nz
            ok = (X >= 0) & (X < gx) & (Y >= 0) & (Y < gy) & (Z >= 0) & (Z < gz) & (taken == 0)
            at = torch.where(ok, (Z * gy + Y) * gx + X, torch.zeros_like(X))
            gid = torch.where(ok, pre[at], torch.zeros_like(at))
            ok &= (gid > 0) & (gid < int(p.maxTotalGrains))
            i = torch.nonzero(ok).flatten()
            at, gid = at[i], gid[i]
            G, dc = self.rot[gid].reshape(-1, 3, 3), self.dc[at]
            half = (torch.einsum("nij,ni->nj", G, -dc).abs().sum(1)).clamp(max=1.5) + self.fs.flatten()[at] * p.rev_fsgrow
            step = torch.tensor([nx, ny, nz], **self.f)
            v = torch.einsum("nij,ni->nj", G, -step - dc)
            won = half - v.abs().sum(1) > 0
            i, gid, G, dc, half, v = i[won], gid[won], G[won], dc[won], half[won], v[won]
            dx, dy, dz = v.T
            left = half - half.clamp(max=1.0)
            rules = (((dx + dy >= 0) & (dx - dy > 0) & (dx + dz > 0) & (dx - dz >= 0), (1, 0, 0)),
                     ((dx + dy <= 0) & (dx - dy < 0) & (dx + dz < 0) & (dx - dz <= 0), (-1, 0, 0)),
                     ((dy + dx > 0) & (dy - dx >= 0) & (dy + dz >= 0) & (dy - dz > 0), (0, 1, 0)),
                     ((dy + dx < 0) & (dy - dx <= 0) & (dy + dz <= 0) & (dy - dz < 0), (0, -1, 0)),
                     ((dz + dx >= 0) & (dz - dx > 0) & (dz + dy > 0) & (dz - dy >= 0), (0, 0, 1)))
            corner = torch.tensor([0.0, 0.0, -1.0], **self.f).expand(len(i), 3).clone()
            todo = torch.ones(len(i), dtype=torch.bool, device=self.dev)
            for cond, unit in rules:
                corner[todo & cond] = torch.tensor(unit, **self.f)
                todo &= ~cond
            centre[i] = dc + step + torch.einsum("nij,nj->ni", G, corner * left[:, None])
            taken[i] = gid
        kept = self.slots[rank, slot]
        kept = torch.where((slot <= zero_to[rank])[:, None], torch.zeros_like(kept), kept)
        value = torch.where((taken > 0)[:, None], centre, kept)
        self.slots[rank, slot] = value
        self.dc[cells] = value
        gr = self.gr.flatten()
        gr[cells] = torch.where(taken > 0, taken, gr[cells])
        self.gr = gr.reshape(self.shape)

    def solid(self):
        return float(self.fs.clamp(max=1.0).sum() / self.fs.numel())

    def field(self, name):
        """The halo'd host array that a download gives."""
        if name == "temperature":
            T = self.temperature(self.ts, halo=True)
            gz, gy, gx = self.shape
            return T.expand(gz + 2, gy + 2, gx + 2).cpu().numpy().copy()
        out = np.full(tuple(n + 2 for n in self.shape), self.p.Cinit if name in ("ce", "cl") else 0.0)
        out[1:-1, 1:-1, 1:-1] = getattr(self, name).cpu().numpy()
        return out


def _exact_adjoint(case, seed):
    d = _inputs(case, seed)
    other = _Run(d, (1.2, 0.9))
    sim = _Run(d)
    for _ in range(case["warm"]):
        other.step()
        sim.step()
    tape = []
    for _ in range(case["steps"]):
        other.step()
        old, T, branch = sim.step()
        tape.append((old if not tape else None, T, branch))
    loss = {}
    leaf = {k: torch.tensor(v, requires_grad=True, **sim.f) for k, v in (("Dliq", sim.p.Dliq), ("k", sim.p.part_coef))}
    dtx = sim.p.ts_delt / (sim.p.cellSize * sim.p.cellSize)
    for name, (a, b) in (("loss", (1.0, 1.0)), ("trial", (1.02, 0.99))):
        par = dict(sim.par, rl=leaf["Dliq"] * a * dtx, dxt=leaf["Dliq"] * a * dtx, k=leaf["k"] * b)
        ce, cl, fs = tape[0][0]
        with torch.set_grad_enabled(name == "loss"):
            for _, T, branch in tape:
                ce, cl, fs, _ = sim.update(ce, cl, fs, T, par, branch)
            loss[name] = 0.5 * ((ce - other.ce) ** 2).sum()
    loss["loss"].backward()
    return {"loss": float(loss["loss"].detach()), "Dliq": float(leaf["Dliq"].grad), "part_coef": float(leaf["k"].grad),
            "gibbs": None, "trial": float(loss["trial"])}


def exact(case, seed):
    if case.get("curv"):
        return None  # a tip's curvature rests on acos and on which components are exactly zero
    if case["kind"] == "adjoint":
        cells = case["nx"] * case["ny"] * case["nz"]
        return _exact_adjoint(case, seed) if cells * case["steps"] < 4e7 else None
    if case["kind"] == "ensemble":
        if case["domains"] > 8:
            return None  # one domain after another takes too long
        runs = [_Run(d) for d in _members(case, seed)]
        for sim in runs:
            for _ in range(case["warm"] + case["steps"]):
                sim.step()
        return {"fs_fraction": np.array([sim.solid() for sim in runs]),
                "ce": np.concatenate([sim.field("ce").ravel() for sim in runs]), "gr": None}
    sim = _Run(_inputs(case, seed))
    for _ in range(case["warm"]):
        sim.step()
    fractions = []
    for n in range(1, case["steps"] + 1):
        sim.step()
        if n % case["read"] == 0 or n == case["steps"]:
            fractions.append(sim.solid())
    out = {"fs_fraction": np.array(fractions), "solute": float(sim.ce.sum())}
    for f in case["fields"].split(","):
        out[f] = None if f == "gr" else sim.field(f)
    return out
