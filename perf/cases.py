"""Performance cases: what a user of this framework has it do, and how large that is.

Every case goes through the public Python calls (Problem, Shot, Batch, Server).  The kinds:

* ``run``: a kept shot, advanced by ``steps`` time steps a pass, its detector traces of these steps, the
  running DFT and an Ez slice read back after them -- how a program follows a long shot, and how the
  reference's driver does (2-D slices every 2000 steps).  The shot starts in mid-run (waves everywhere in the
  grid), not in an empty grid.  When its steps are used up the program goes on with the next shot.
* ``ini``: the same for a shot of a Settings.ini (material-ID medium, 10-50 GHz array, wave-front tracker lines).
* ``whole``: a parameter sweep's inner call: create a shot from a host setup, run it, read it, release it.
* ``batch``: uneven shots admitted to one batch, advanced together, their DFTs and traces read after each block.
* ``serve``: requests submitted to the serving loop, stepped until all are done, their results popped.

Sizes come from the repository's own workloads: the 256 x 192 shot of the smoke test, the plain 512^2 shot, the
8192^2 production shot, the default Settings.ini (500 x 3000 cells, 21 tracker lines), the mixed-size sample of
the benchmark's batched and serving legs (sides from 512 up, CPML 10 to 32).
"""
import math
import os
import random
import tempfile

import numpy as np
import torch

import fdtd_2d_gb300 as F

STORES = {"f32": F.STORE_F32, "f16": F.STORE_F16, "bf16": F.STORE_BF16}


def listed():
    return [
        # the smallest call in use: the smoke test's shot, a probe of a setup before a sweep
        {"name": "run_256x192", "kind": "run", "nx": 256, "ny": 192, "npml": 10, "steps": 2000, "store": "f32", "plasma": 1, "array": 1},
        # the plain 512^2 shot (point source, linear slab, 10-cell CPML)
        {"name": "run_512", "kind": "run", "nx": 512, "ny": 512, "npml": 10, "steps": 2000, "store": "f32", "plasma": 1, "array": 1},
        # a ragged grid with a random-field plasma: an odd member of the mixed-size sample
        {"name": "run_777x1301", "kind": "run", "nx": 777, "ny": 1301, "npml": 17, "steps": 1500, "store": "f32", "plasma": 3, "array": 7},
        # mid-size shots of the mixed sample
        {"name": "run_2048", "kind": "run", "nx": 2048, "ny": 2048, "npml": 32, "steps": 1000, "store": "f32", "plasma": 2, "array": 16},
        {"name": "run_2300x1531_bf16", "kind": "run", "nx": 2300, "ny": 1531, "npml": 24, "steps": 400, "store": "bf16", "plasma": 2, "array": 9},
        {"name": "run_4096_f16", "kind": "run", "nx": 4096, "ny": 4096, "npml": 32, "steps": 600, "store": "f16", "plasma": 2, "array": 16},
        # the production shot
        {"name": "run_8192", "kind": "run", "nx": 8192, "ny": 8192, "npml": 32, "steps": 600, "store": "f32", "plasma": 2, "array": 16},
        # the default Settings.ini: the reference's own workload
        {"name": "ini_500x3000", "kind": "ini", "imax": 250, "jmax": 1500, "steps": 2000, "wall": 0},
        # a Settings.ini with the steel wall (its coefficients differ: the material-ID medium)
        {"name": "ini_wall_500x1200", "kind": "ini", "imax": 250, "jmax": 600, "steps": 1000, "wall": 1},
        # one point of a parameter sweep, from host arrays to host results
        {"name": "whole_1024", "kind": "whole", "nx": 1024, "ny": 1024, "npml": 20, "steps": 1200, "store": "f32", "plasma": 2, "array": 8},
        # the batched leg's mix, at its smaller sides
        {"name": "batch_12", "kind": "batch", "shots": 12, "lo": 512, "hi": 1800, "steps": 128, "mix": 1},
        # a request of a frequency sweep through the serving loop
        {"name": "serve_8x700", "kind": "serve", "shots": 8, "lo": 700, "hi": 700, "steps": 500, "mix": 2},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "run", "ini", "whole", "batch", "serve"])
    if kind == "batch":
        lo = _log(rng, 400, 900)
        return {"kind": kind, "shots": rng.randint(4, 16), "lo": lo, "hi": _log(rng, lo + 100, 1800), "steps": rng.randint(48, 160), "mix": rng.randint(1, 10**6)}
    if kind == "serve":
        lo = _log(rng, 400, 900)
        return {"kind": kind, "shots": rng.randint(4, 12), "lo": lo, "hi": lo, "steps": rng.randint(300, 700), "mix": rng.randint(1, 10**6)}
    if kind == "ini":
        return {"kind": kind, "imax": _log(rng, 150, 400), "jmax": _log(rng, 400, 1500), "steps": rng.randint(500, 2000), "wall": rng.choice([0, 0, 1])}
    cells = math.exp(rng.uniform(math.log(4e4), math.log(2e6 if kind == "whole" else 4e7)))
    aspect = math.exp(rng.uniform(-math.log(3), math.log(3)))
    nx, ny = max(160, int(math.sqrt(cells * aspect))), max(160, int(math.sqrt(cells / aspect)))
    store = "f32" if kind == "whole" else rng.choice(["f32", "f32", "f32", "f16", "bf16"])
    steps = int(min(2000, max(300, 3.5e10 / (nx * ny))))
    return {"kind": kind, "nx": nx, "ny": ny, "npml": rng.randint(10, 32), "steps": rng.randint(steps // 2, steps) if store != "bf16" else rng.randint(200, 400),
            "store": store, "plasma": rng.choice([1, 2, 2, 3]), "array": rng.randint(1, 16)}


# ---- inputs -----------------------------------------------------------------------------------------------------------

#: steps of a kept shot: as many as the program reads back before it goes on with the next one
LONG = {"run": 60000, "ini": 33568, "batch": 16000}


def _spec(case, rng, n_steps):
    """A shot of the repository's synthetic workloads: array of `array` elements, plasma profile 1 (slab), 2 (tanh) or 3 (tanh x random field)."""
    nx, ny, P, m = case["nx"], case["ny"], case["npml"], case["array"]
    dx = 0.25e-3 if nx * ny > 1 << 20 else 0.5e-3
    freq = rng.uniform(20e9, 30e9) if dx > 0.3e-3 else rng.uniform(40e9, 55e9)
    peak = rng.uniform(1e19, 2.8e19)
    i0 = P + max(4, min(32, nx // 16))
    j0 = ny // 2 - (m - 1) * 5 // 2
    return F.default_spec(
        nx=nx, ny=ny, npml=P, n_steps=n_steps, dx=dx, dy=dx, courant=0.97, profile=case["plasma"], ne_peak=peak,
        x_lo=nx // 2, x_hi=nx - P, x_center=nx * rng.uniform(0.5, 0.7), width=nx * rng.uniform(0.06, 0.12), grf_rms=0.05, grf_corr=min(40, nx / 16),
        seed=rng.randint(1, 10**6), nu=rng.choice([1e9, 2e9]), n_elem=m, src_i=i0, src_j=j0, src_di=0, src_dj=5, freq=freq, steer_deg=rng.uniform(-15, 15),
        pulse=1, pulse_width=0.2e-9, n_det=m, det_i=i0 + 2, det_j=j0, det_di=0, det_dj=5, record_traces=1, dft_freq=freq, storage=STORES[case.get("store", "f32")],
        field_max=4.0)


INI = """[grid]
Use_Exp_time = 0
Imax = {imax}
Jmax = {jmax}
Max_time = {n}
ds = 0.5
dt_coef = 0.5
Isource = {isrc}
Jsource = 20
Idetect = {isrc}
Jdetect = 24
[AESA]
SIsize = 40
SIdelta = 5
SPAngle = {angle}
DIsize = 40
DIdelta = 5
[PulseParam]
Chirp = 0
FreqA = {freq}
Fronts = 600
Plato = 1200
Pulse_amp = 1881
[medium]
Build = 1
Icen = {isrc}
Jcen = {jcen}
Radius = {radius}
ne0 = {ne0}
[KameraConf]
DrawWall = {wall}
WallPos = {wallpos}
[RC_calc]
Iline = {isrc}
LIsize = 100
LIdelta = 5
Rlevel = 0.07
"""


def _ini(case, rng):
    text = INI.format(imax=case["imax"], jmax=case["jmax"], n=LONG["ini"], isrc=case["imax"] // 2, jcen=case["jmax"] * 2 // 3, radius=case["imax"] // 3,
                      ne0="%.4e" % rng.uniform(2e19, 5.5e19), angle="%.3f" % rng.uniform(-8, 8), freq="%.3f" % rng.uniform(30, 40), wall=case["wall"],
                      wallpos=case["jmax"] * 18 // 10)
    fd, path = tempfile.mkstemp(suffix=".ini")
    with os.fdopen(fd, "w") as f:
        f.write(text)
    try:
        return F.Problem.from_ini(path)
    finally:
        os.unlink(path)


def _waves(nx, ny, rng):
    """Ez in mid-run: plane waves of 12 to 60 cells, of amplitude up to 1 in all."""
    k = 6
    x, y = np.empty((k, nx), np.float32), np.empty((ny, k), np.float32)
    for q in range(k):
        for v, n in ((x[q], nx), (y[:, q], ny)):
            v[:] = np.cos(2 * math.pi * (np.arange(n) / rng.uniform(12, 60) + rng.random()))
    y *= 1.0 / k
    return y @ x


def _members(case, rng):
    """The shots of a batch or of a request: their grids from the case, the rest from the seed."""
    size = random.Random(case["mix"])
    out = []
    for _ in range(case["shots"]):
        nx = max(160, _log(size, case["lo"], case["hi"]))
        ny = nx if case["lo"] == case["hi"] else max(160, int(nx * math.exp(size.uniform(-math.log(2), 0))))
        out.append({"nx": nx, "ny": ny, "npml": size.randint(16, 32), "plasma": 2, "array": size.randint(4, 12)})
    n = case["steps"] if case["kind"] == "serve" else LONG["batch"]
    return [F.Problem.from_spec(_spec(c, rng, n)) for c in out]


def _inputs(case, seed):
    """(problems, the Ez that a kept shot starts with)"""
    rng = random.Random(1000003 * seed + 17)
    kind = case["kind"]
    if kind in ("batch", "serve"):
        return _members(case, rng), None
    if kind == "ini":
        return [_ini(case, rng)], None
    p = F.Problem.from_spec(_spec(case, rng, case["steps"] if kind == "whole" else LONG["run"]))
    return [p], _waves(p.nx, p.ny, rng) if kind == "run" else None


def _begin(state):
    """The handle that the program keeps over its passes."""
    kind, problems = state["kind"], state["problems"]
    if kind in ("run", "ini"):
        state["shot"] = F.Shot(problems[0])
        if state["ez"] is not None:
            state["shot"].write_field("ez", state["ez"])
    elif kind == "batch":
        state["batch"] = F.Batch()
        state["ids"] = [state["batch"].add(p) for p in problems]
    elif kind == "serve":
        state["server"] = F.Server()


def prepare(case, seed):
    problems, ez = _inputs(case, seed)
    state = {"kind": case["kind"], "steps": case["steps"], "problems": problems, "ez": ez}
    _begin(state)
    return state


def run(state):
    kind, k = state["kind"], state["steps"]
    if kind in ("run", "ini"):
        shot = state["shot"]
        n = shot.step
        if n + k > shot.n_steps:
            shot.close()
            state["ez"] = None   # the next shot starts from rest
            _begin(state)
            shot, n = state["shot"], 0
        shot.run(n + 1, n + k)
        out = {"traces": shot.traces(n + 1, n + k)["det_ez"], "ez": shot.read_field("ez")}
        if kind == "run":
            out["dft"] = shot.dft()
        else:
            out["rc"] = shot.rc(n + 1, n + k)
        return out
    if kind == "whole":
        with F.Shot(state["problems"][0]) as shot:
            shot.run(1, k)
            return {"traces": shot.traces()["det_ez"], "dft": shot.dft(), "ez": shot.read_field("ez")}
    if kind == "batch":
        b, ids = state["batch"], state["ids"]
        n = b.step(ids[0])
        if n + k > LONG["batch"]:
            for i in ids:
                b.remove(i)
            ids = state["ids"] = [b.add(p) for p in state["problems"]]
            n = 0
        b.run(k)
        b.synchronize()
        members = [b.shot(i) for i in ids]
        return {"traces": [m.traces(n + 1, n + k)["det_ez"] for m in members], "dft": [m.dft() for m in members]}
    server, problems = state["server"], state["problems"]
    for tag, p in enumerate(problems):
        server.submit(p, tag)
    got = {}
    while len(got) < len(problems):
        server.step()
        while (r := server.pop()) is not None:
            got[r["tag"]] = r
    return {"traces": [got[t]["det_ez"] for t in range(len(problems))], "dft": [got[t]["dft"] for t in range(len(problems))]}


def work(case):
    """The state (Ez, Hx, Hy, Jz) read and written once and the drive map read once a pass; an update of a cell takes 20 operations
    (Hx 4, Hy 4, Jz 3, Ez 9)."""
    if case["kind"] in ("batch", "serve"):
        problems = _members(case, random.Random(1))
        cells = sum(p.nx * p.ny for p in problems)
    elif case["kind"] == "ini":
        cells = 4 * case["imax"] * case["jmax"]
    else:
        cells = case["nx"] * case["ny"]
    per = 36 if case.get("store", "f32") == "f32" else 18
    return {"bytes": per * cells, "flops": 20 * cells * case["steps"]}


# ---- the same in 64 bits ----------------------------------------------------------------------------------------------

def _points(p, n):
    return [(p[k].j, p[k].i) for k in range(n)]


class _Exact:
    """The TMz update with convolutional PML, Drude current, soft sources and detectors on the arrays of a setup, in FP64."""

    def __init__(self, problem):
        s = problem.setup
        self.dev = dev = "cuda" if torch.cuda.is_available() else "cpu"
        nx, ny, P = self.nx, self.ny, self.P = s.nx, s.ny, s.npml
        self.s = s

        def t(a):
            return torch.from_numpy(np.asarray(a, np.float64)).to(dev)

        def tab(name, n):
            return t(problem.array(name, n))

        self.dex, self.dhx = tab("den_ex", nx - 1)[None, :], tab("den_hx", nx - 1)[None, :]
        self.dey, self.dhy = tab("den_ey", ny - 1)[:, None], tab("den_hy", ny - 1)[:, None]
        # strips of depth P - 1: rows (columns) 0.. and ..end, the second strip's tables run from the outer edge inwards
        self.strips = {}
        for f, a, d in (("be", "x", s.dx), ("bh", "x", s.dx), ("be", "y", s.dy), ("bh", "y", s.dy)):
            c = "c" + f[1]
            n = P if f == "be" else P - 1
            cut = slice(1, P) if f == "be" else slice(0, P - 1)
            for side in (1, 2):
                b, cc = tab("%s_%s_%d" % (f, a, side), n)[cut], tab("%s_%s_%d" % (c, a, side), n)[cut] / float(np.float32(d))
                if side == 2:
                    b, cc = b.flip(0), cc.flip(0)
                shape = (-1, 1) if a == "y" else (1, -1)
                size = (P - 1, nx) if a == "y" else (ny, P - 1)
                self.strips[f, a, side] = (b.reshape(shape), cc.reshape(shape), torch.zeros(size, dtype=torch.float64, device=dev))
        beta = s.jz_coef * s.dt / (1 + 0.5 * s.nu * s.dt)
        self.ja = (1 - 0.5 * s.nu * s.dt) / (1 + 0.5 * s.nu * s.dt)
        if s.medium == F.MEDIUM_UNIFORM:
            self.da1 = self.da2 = float(s.da)
            self.db1 = self.db2 = float(s.db)
            self.ca, self.cb, self.keep = float(s.ca), float(s.cb), None
            ne = t(problem.array("ne", nx * ny)).reshape(ny, nx) if s.ne else None
        else:
            ids = [torch.from_numpy(problem.array(n, nx * ny, np.int64)).to(dev).reshape(ny, nx) for n in ("id1", "id2", "id3")]
            da, db, ca, cb, mne = (tab(n, s.n_materials) for n in ("mat_da", "mat_db", "mat_ca", "mat_cb", "mat_ne"))
            self.da1, self.db1, self.da2, self.db2 = da[ids[0]], db[ids[0]], da[ids[1]], db[ids[1]]
            self.ca, self.cb, ne = ca[ids[2]], cb[ids[2]], mne[ids[2]]
            self.keep = (ids[2] != 1).double()[1:-1, 1:-1]
        if ne is None:
            self.kp = None
        else:
            ne = ne[1:-1, 1:-1]
            self.kp = torch.where(ne > 0, beta * ne, torch.zeros_like(ne))
            self.jd = torch.where(ne > 0, torch.full_like(ne, self.ja), torch.ones_like(ne))
        self.ez, self.hx, self.hy, self.jz = (torch.zeros((ny, nx), dtype=torch.float64, device=dev) for _ in range(4))

    def at(self, c, rows, cols):
        return c[rows, cols] if isinstance(c, torch.Tensor) else c

    def psi(self, key, rows, cols, diff, coef, field):
        """One strip: psi = b psi + c/d diff, field += coef psi."""
        b, c, psi = self.strips[key]
        v = psi[:, cols] if key[1] == "y" else psi[rows, :]
        v.mul_(b).add_(diff * c)
        field[rows, cols] += self.at(coef, rows, cols) * v

    def steps(self, n_steps, first):
        s, P, nx, ny = self.s, self.P, self.nx, self.ny
        ez, hx, hy, jz = self.ez, self.hx, self.hy, self.jz
        h, e = slice(0, -1), slice(1, -1)
        lo_h, hi_h, lo_e, hi_e = slice(0, P - 1), lambda n: slice(n - P, n - 1), slice(1, P), lambda n: slice(n - P, n - 1)
        src, det = _points(s.src, s.n_src), _points(s.det, s.n_det)
        sj, si = (torch.tensor([q[k] for q in src], device=self.dev, dtype=torch.long) for k in (0, 1))
        dj, di = (torch.tensor([q[k] for q in det], device=self.dev, dtype=torch.long) for k in (0, 1))
        n = np.arange(first, first + n_steps, dtype=np.float64)
        time = n * s.dt
        chirp = 0.5 * (s.f1 - s.f0) / s.t1 if s.f1 != s.f0 else 0.0
        phase = np.array([s.src_phase_deg[k] for k in range(s.n_src)]) / 360
        x = (chirp * time**2 + s.f0 * time)[:, None] + phase[None, :]
        if s.src_pi in (0.0, math.pi):
            val = np.cos(2 * math.pi * (x - np.floor(x)))
        else:
            val = np.cos(2 * s.src_pi * x)
        env = np.array([s.envelope[int(k)] for k in n], np.float64)
        val = torch.from_numpy(s.src_scale * env[:, None] * val).to(self.dev)
        trace = torch.zeros((n_steps, s.n_det), dtype=torch.float64, device=self.dev)
        for q in range(n_steps):
            d = ez[h, h] - ez[1:, h]
            if not isinstance(self.da1, float):
                hx[h, h] = self.da1[h, h] * hx[h, h] + self.db1[h, h] * (d * self.dhy)
            else:
                hx[h, h].mul_(self.da1).add_(d * self.dhy, alpha=self.db1)
            self.psi(("bh", "y", 1), lo_h, h, d[lo_h, :], self.db1, hx)
            self.psi(("bh", "y", 2), hi_h(ny), h, d[ny - P:ny - 1, :], self.db1, hx)
            d = ez[h, 1:] - ez[h, h]
            if not isinstance(self.da2, float):
                hy[h, h] = self.da2[h, h] * hy[h, h] + self.db2[h, h] * (d * self.dhx)
            else:
                hy[h, h].mul_(self.da2).add_(d * self.dhx, alpha=self.db2)
            self.psi(("bh", "x", 1), h, lo_h, d[:, lo_h], self.db2, hy)
            self.psi(("bh", "x", 2), h, hi_h(nx), d[:, nx - P:nx - 1], self.db2, hy)
            if self.kp is not None:
                jz[e, e].mul_(self.jd).addcmul_(self.kp, ez[e, e])
            dy, dx = hy[e, e] - hy[e, :-2], hx[:-2, e] - hx[e, e]
            curl = (dy * self.dex[:, 1:]).addcmul_(dx, self.dey[1:]).sub_(jz[e, e])
            ez[e, e] = self.at(self.ca, e, e) * ez[e, e] + self.at(self.cb, e, e) * curl
            if self.keep is not None:
                ez[e, e] *= self.keep
            self.psi(("be", "x", 1), e, lo_e, dy[:, lo_h], self.cb, ez)
            self.psi(("be", "x", 2), e, hi_e(nx), dy[:, nx - P - 1:nx - 2], self.cb, ez)
            self.psi(("be", "y", 1), lo_e, e, dx[lo_h, :], self.cb, ez)
            self.psi(("be", "y", 2), hi_e(ny), e, dx[ny - P - 1:ny - 2, :], self.cb, ez)
            if len(src):
                ez.index_put_((sj, si), -val[q], accumulate=True)
            trace[q] = ez[dj, di]
        out = {"traces": trace, "ez": ez}
        if s.dft_freq > 0:
            ph = s.dft_freq * s.dt * n
            ph = 2 * math.pi * (ph - np.floor(ph))
            w = torch.from_numpy(np.stack([np.cos(ph), -np.sin(ph)])).to(self.dev)
            re, im = (w @ trace).cpu().numpy()
            out["dft"] = re + 1j * im
        return out


def _covered(s):
    """Whether the reference's launches reach every cell: where they do not, it leaves cells out."""
    X, Y, Q = s.nx, s.ny, s.npml - 1
    need = [(Y - 1) * (X - 1), Q * (X - 1), Y * (X - 1), Y * Q, (Y - 2) * (X - 2), (Y - 2) * (X - 2), (Y - 2) * Q, Q * (X - 2)]
    return all(c == 0 or c >= n for c, n in zip(s.cover, need))


def exact(case, seed):
    problems, ez = _inputs(case, seed)
    if not all(_covered(p.setup) for p in problems):
        return None
    if sum(p.nx * p.ny for p in problems) * case["steps"] > 9e10:
        return None
    got = []
    for p in problems:
        x = _Exact(p)
        if ez is not None:
            x.ez.copy_(torch.from_numpy(ez))
        got.append(x.steps(case["steps"], 1))
    if case["kind"] in ("run", "whole"):
        return {k: got[0][k] for k in ("traces", "ez", "dft")}
    if case["kind"] == "ini":
        return {"traces": got[0]["traces"], "ez": got[0]["ez"], "rc": None}
    return {"traces": [g["traces"] for g in got], "dft": [g["dft"] for g in got]}
