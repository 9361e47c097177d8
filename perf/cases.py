"""Performance cases of the FDTD engine: whole simulations through the public
entry points (Engine, Batch, Server), as a program that uses the framework
runs them: reset, iterate, read the samples and the final fields.

A case is a dict of plain values:

    kind     run    one simulation on one engine
             batch  a parameter sweep: `jobs` simulations in one Batch
             serve  `jobs` requests through a Server, operator builds included
    media    bricks       dielectric bricks and a 50 ohm port on a uniform mesh
             dispersive   Drude and Lorentz bricks on a graded mesh
             multipole    materials with several poles, electric and magnetic
             channel      a plane wave through a double-negative Drude slab
    nx ny nz cells per axis;  pml: UPML layers (0: PEC walls);  mur: Mur faces
    steps    timesteps;  fresh: the engine is made (operator uploaded) in the
             pass;  freqs: frequency-domain probe frequencies;  frames: field
             dumps taken on the way;  rlc: lumped RLC elements

The geometry (bricks and their materials) comes from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from wipems_gb300 import Batch, CompressedOperator, Engine, Operator, Server, scenes
from wipems_gb300.fdtd import BC_MUR, BC_PEC, BC_PML, Scene

EPS0 = 8.85418781762e-12
MUE0 = 1.256637062e-6


def _case(name, kind="run", media="bricks", n=(32, 32, 32), steps=500, pml=0, **kv):
    c = dict(name=name, kind=kind, media=media, nx=n[0], ny=n[1], nz=n[2], steps=steps, pml=pml, mur=False,
             fresh=False, freqs=0, frames=0, rlc=0, jobs=1)
    c.update(kv)
    return c


def listed():
    return [
        # the smallest simulation of the reference's test suite: the mesh of the cavity resonance test
        _case("cavity", n=(25, 10, 31), steps=2000),
        # the plain 64^3 PEC box
        _case("p64", n=(64, 64, 64), steps=1000),
        # the quasi-2D double-negative Drude slab example: Mur, PMC and PEC walls, a long thin grid
        _case("channel", media="channel", n=(20, 3, 1000), steps=1000),
        # a small antenna-like run: ragged UPML grid with frequency-domain port sums (S-parameters)
        _case("sparam_small", n=(47, 33, 61), steps=800, pml=8, freqs=32),
        # one job of a sweep over PEC boxes, end to end: engine made, run, read, closed
        _case("sweep_pec", n=(131, 97, 75), steps=1000, fresh=True),
        # a field monitor: E and H dumps on the way through a mid-size UPML run
        _case("monitor_upml", n=(150, 118, 101), steps=600, pml=8, frames=4),
        # Mur walls and lumped RLC elements beside the port
        _case("mur_rlc", n=(112, 96, 128), steps=500, mur=True, rlc=3),
        # multi-pole electric and magnetic materials on a graded mesh
        _case("multipole", media="multipole", n=(84, 76, 92), steps=400, pml=8),
        # the dispersive graded-mesh workload (192^3 cells)
        _case("d192", media="dispersive", n=(192, 192, 192), steps=800, pml=8),
        # the headline workload: 256^3 cells, UPML-8, 40 bricks, 1000 timesteps
        _case("l256", n=(256, 256, 256), steps=1000, pml=8),
        # a parameter sweep in one batch: uneven jobs, half PEC and half UPML
        _case("batch12", kind="batch", n=(48, 104, 160), steps=400, pml=8, jobs=12),
        # a burst of requests through the server, each until its energy has decayed by 40 dB
        _case("serve16", kind="serve", n=(32, 64, 128), steps=4000, pml=8, jobs=16),
    ]


def draw(rng):
    def edge(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    what = rng.choice(["run", "run", "run", "run", "dispersive", "multipole", "channel", "batch"])
    steps = edge(200, 1200)
    if what == "channel":
        return _unnamed(_case("", media="channel", n=(edge(8, 40), edge(3, 8), edge(200, 1500)), steps=steps))
    if what == "batch":
        lo = edge(32, 64)
        return _unnamed(_case("", kind="batch", n=(lo, lo + 20, edge(lo + 30, 160)), steps=edge(100, 400), pml=8,
                              jobs=rng.randint(3, 12)))
    if what in ("dispersive", "multipole"):
        top = 192 if what == "dispersive" else 110
        return _unnamed(_case("", media=what, n=tuple(edge(40, top) for _ in range(3)), steps=min(steps, 600), pml=8))
    wall = rng.choice(["pec", "upml", "upml", "mur"])
    n = tuple(edge(32, 256) for _ in range(3))
    kv = dict(pml=8 if wall == "upml" else 0, mur=wall == "mur", fresh=rng.random() < 0.3)
    if rng.random() < 0.3:
        kv["freqs"] = edge(4, 64)
    if rng.random() < 0.2:
        kv["frames"] = rng.randint(1, 4)
    if rng.random() < 0.2:
        kv["rlc"] = rng.randint(1, 4)
    return _unnamed(_case("", n=n, steps=steps, **kv))


def _unnamed(c):
    del c["name"]
    return c


# ------------------------------------------------------------------ scenes
def _boxes(rng, lines, margin, count, emin, emax):
    out = []
    for _ in range(count):
        a, b = [], []
        for L in lines:
            cells = len(L) - 1
            e = int(rng.integers(emin, max(emin, min(emax, cells - 2 * margin)) + 1))
            s = int(rng.integers(margin, max(margin, cells - margin - e) + 1))
            a.append(L[s])
            b.append(L[min(s + e, cells)])
        out.append((a, b))
    return out


def _port(s, lines):
    c = [len(L) // 2 for L in lines]
    s.add_lumped_port([lines[0][c[0]], lines[1][c[1]], lines[2][c[2] - 2]],
                      [lines[0][c[0] + 1], lines[1][c[1] + 1], lines[2][c[2] + 2]], 2, 50.0, priority=100000)


def _scene(case, seed):
    n = (case["nx"], case["ny"], case["nz"])
    rng = np.random.default_rng(seed)
    if case["media"] == "channel":
        mx = (np.arange(n[0] + 1) - n[0] / 2) * 0.5
        my = (np.arange(n[1] + 1) - n[1] / 2) * 0.5
        mz = (np.arange(n[2] + 1) - n[2] / 2) * 0.5
        s = Scene(mx, my, mz, 1e-3)
        s.set_boundary([1, 1, BC_PEC, BC_PEC, BC_MUR, BC_MUR], [0] * 6)  # 1: PMC
        s.set_gauss_excite(0.0, 10e9, case["steps"])
        s.set_oversampling(10)
        s.add_excitation([mx[0], my[0], mz[2]], [mx[-1], my[-1], mz[2]], [0, 1, 0], priority=0)
        f0, tau = float(rng.uniform(4e9, 6e9)), 5e-9
        q = n[2] // 4
        s.add_lorentz([mx[0], my[0], mz[q]], [mx[-1], my[-1], mz[-1 - q]], plasma_f=[f0], relax_t=[tau],
                      mue_plasma_f=[f0], mue_relax_t=[tau], priority=10)
        for k in (n[2] // 8, n[2] // 2, n[2] - n[2] // 8):
            s.add_probe([mx[n[0] // 2], my[0], mz[k]], [mx[n[0] // 2], my[-1], mz[k]], 0)
        return s
    graded = case["media"] in ("dispersive", "multipole")
    # the mesh grading depends on the size alone, so the timestep and the number of samples do too
    mesh = np.random.default_rng(11)
    lines = [scenes.graded_lines(c, mesh) if graded else scenes.uniform_lines(c, 0.5) for c in n]
    s = Scene(*lines, 1e-3)
    pml = case["pml"]
    s.set_boundary([BC_PML if pml else BC_MUR if case["mur"] else BC_PEC] * 6, [pml] * 6)
    f0 = 6e9 if graded else 10e9
    s.set_gauss_excite(f0, f0, case["steps"])
    m, prio = pml + 1, 10
    small = min(n)
    if case["media"] == "bricks":
        count = max(2, min(40, int(n[0] * n[1] * n[2] / 4e5)))
        for a, b in _boxes(rng, lines, m, count, max(2, small // 32), max(3, small // 4)):
            s.add_material(a, b, eps_r=float(rng.uniform(1, 12)), kappa=float(10 ** rng.uniform(-4, 0)), priority=prio)
            prio += 1
    elif case["media"] == "dispersive":  # about 40 % of the volume, Drude and single-pole Lorentz
        for k, (a, b) in enumerate(_boxes(rng, lines, m, 40, max(2, small // 16), max(3, small // 4))):
            if k % 8 < 5:
                s.add_lorentz(a, b, plasma_f=[2e9], relax_t=[1.0 / float(10 ** rng.uniform(7, 8))], pole_f=[0.0],
                              priority=prio)
            else:
                fl = float(rng.uniform(2e9, 20e9))
                s.add_lorentz(a, b, eps_r=float(rng.uniform(2, 4)), plasma_f=[fl * math.sqrt(float(rng.uniform(1, 5)))],
                              relax_t=[1.0 / float(10 ** rng.uniform(8, 9))], pole_f=[fl], priority=prio)
            prio += 1
    else:
        for k, (a, b) in enumerate(_boxes(rng, lines, m, 6, max(2, small // 8), max(3, small // 3))):
            f = float(rng.uniform(4e9, 9e9))
            if k % 3 == 0:
                s.add_lorentz(a, b, eps_r=2.0, plasma_f=[f, 1.5 * f, 0.7 * f], relax_t=[1e-9, 2e-9, 0.5e-9],
                              pole_f=[0.0, 7e9, 11e9], priority=prio)
            elif k % 3 == 1:
                s.add_lorentz(a, b, eps_r=3.0, plasma_f=[f, 8e9], relax_t=[1e-9, 1e-9], pole_f=[6e9, 0.0],
                              mue_plasma_f=[0.0, 4e9], mue_relax_t=[0.0, 1e-9], priority=prio)
            else:
                s.add_lorentz(a, b, eps_r=1.5, plasma_f=[f], relax_t=[2e-9], priority=prio)
            prio += 1
    c = [len(L) // 2 for L in lines]
    for k in range(case["rlc"]):
        x, y = lines[0][c[0] - 5 + 3 * k], lines[1][c[1] + 4]
        s.add_lumped_rlc([x, y, lines[2][c[2] - 2]], [x, y, lines[2][c[2] + 1]], 2, R=20.0 + 10 * k, L=2e-9,
                         Cap=0.5e-12, series=k % 2 == 0, caps=False, priority=90000)
    _port(s, lines)
    return s


def _sizes(case):
    """Uneven grids between the case's smallest and largest edge: the size
    of job k depends on k alone, so a case costs the same for every seed."""
    lo, hi = case["nx"], case["nz"]
    rng = np.random.default_rng(7)
    return [tuple(int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) for _ in range(3))
            for _ in range(case["jobs"])]


def _job_cases(case):
    out = []
    for k, n in enumerate(_sizes(case)):
        d = dict(case, kind="run", nx=n[0], ny=n[1], nz=n[2], jobs=1)
        if case["kind"] == "batch":
            d["pml"] = case["pml"] if k % 2 else 0
        out.append(d)
    return out


# ----------------------------------------------------------------- prepare
class _State:
    def __init__(self, case):
        self.case = case


def prepare(case, seed):
    st = _State(case)
    if case["kind"] == "serve":
        st.seed = seed
        st.server = Server()
        return st
    if case["kind"] == "batch":
        cops = [CompressedOperator(Operator(_scene(d, seed + 97 * k))) for k, d in enumerate(_job_cases(case))]
        st.engines = [Engine(c, max_timesteps=case["steps"], kernel="tma") for c in cops]
        # the tiling the batch autotuner picks for sweeps of this kind
        st.batch = Batch(st.engines, x_chunk=64, blocks_per_sm=-1, chains=2, graph_steps=32)
        return st
    st.cop = CompressedOperator(Operator(_scene(case, seed)))
    if not case["fresh"]:
        st.engine = _engine(case, st.cop)
    return st


def _engine(case, cop):
    e = Engine(cop, max_timesteps=case["steps"])
    if case["freqs"]:
        e.set_frequencies(np.linspace(1e9, 15e9, case["freqs"]))
    return e


# --------------------------------------------------------------------- run
def _result(e):
    s = e.samples()
    V, I = e.fields()
    return dict(V=V, I=I, ts=s.ts, values=s.values, energy=s.energy)


def run(st):
    case = st.case
    if case["kind"] == "serve":
        ids = [st.server.submit(_scene(d, st.seed + 97 * k), end_crit=1e-4) for k, d in
               enumerate(_job_cases(case))]
        st.server.wait(0)
        out = []
        for j in ids:  # each job's samples, in a table as long as the timestep cap allows
            s = st.server.samples(j)
            rows = np.zeros((case["steps"] // st.server.status(j)["probe_interval"] + 2, 2 + s.values.shape[1]))
            rows[:len(s.ts)] = np.column_stack([s.ts, s.energy, s.values])
            out.append(rows)
            st.server.release(j)
        return out
    if case["kind"] == "batch":
        for e in st.engines:
            e.reset()
        st.batch.iterate(case["steps"])
        return [list(_result(e).values()) for e in st.engines]
    if case["fresh"]:
        e = _engine(case, st.cop)
    else:
        e = st.engine
        e.reset()
    frames = []
    if case["frames"]:
        for _ in range(case["frames"]):
            e.iterate(case["steps"] // case["frames"])
            frames.append(e.dump_field("E", "cell"))
            frames.append(e.dump_field("H", "node", step=(2, 2, 2)))
        e.iterate(case["steps"] - e.num_timesteps)
    else:
        e.iterate(case["steps"])
    out = _result(e)
    if frames:
        out["frames"] = frames
    if case["freqs"]:
        out["fd"] = e.fd_results()[0]
    if case["fresh"]:
        e.close()
    return out


# -------------------------------------------------------------------- work
def _nodes(case):
    return (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1)


def work(case):
    """One pass: the operator (a 16-bit index per node and half-step) read
    once and the fields written once; 36 operations per node and timestep,
    30 more on UPML nodes, 21 more on the dispersive share."""
    if case["kind"] != "run":
        jobs = _job_cases(case)
        if case["kind"] == "serve":  # the energy decides where a job stops: a few hundred timesteps at least
            jobs = [dict(d, steps=400) for d in jobs]
        parts = [work(d) for d in jobs]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n = _nodes(case)
    inner = (case["nx"] + 1 - 2 * case["pml"]) * (case["ny"] + 1 - 2 * case["pml"]) * (case["nz"] + 1 - 2 * case["pml"])
    flops = 36.0 * n + (30.0 * (n - max(inner, 0)) if case["pml"] else 0.0)
    if case["media"] != "bricks":
        flops += 21.0 * 0.4 * n
    return {"bytes": 28.0 * n, "flops": flops * case["steps"]}


# ------------------------------------------------------------------- exact
# The stepping in 64 bits: the operator's coefficient arrays and lists (the
# engine's input) stepped by plain torch in double.
def _arr(p, shape, dtype=np.float64):
    return np.ctypeslib.as_array(p, shape=(int(np.prod(shape)),)).reshape(shape).astype(dtype)


class _Exact:
    def __init__(self, op):
        self.op, self.d = op, op.desc
        d = self.d
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.N = N = op.num_lines
        shape = (3,) + tuple(N)
        self.vv, self.vi, self.ii, self.iv = (self.t(_arr(getattr(d, k), shape)) for k in ("vv", "vi", "ii", "iv"))
        self.V = torch.zeros(shape, dtype=torch.float64, device=self.dev)
        self.I = torch.zeros_like(self.V)
        self.slabs = []
        for k in range(d.num_upml):
            u = d.upml[k]
            s, n = list(u.start), list(u.num_lines)
            sl = (slice(None),) + tuple(slice(a, a + b) for a, b in zip(s, n))
            c = [self.t(_arr(getattr(u, w), (3, *n))) for w in ("vv", "vvfo", "vvfn", "ii", "iifo", "iifn")]
            if c[0].numel():
                self.slabs.append((sl, c, [torch.zeros_like(c[0]), torch.zeros_like(c[0])]))
        self.ade = []
        for k in range(d.num_ade_orders):
            a = d.ade[k]
            if not a.count:
                continue
            pos = [self.t(_arr(a.pos[q], (a.count,), np.int64)) for q in range(3)]
            lin = (pos[0] * N[1] + pos[1]) * N[2] + pos[2]
            for half, on, lor, names in ((0, a.volt_on, a.volt_lor_on, ("v_int", "v_ext", "v_lor")),
                                         (1, a.curr_on, a.curr_lor_on, ("i_int", "i_ext", "i_lor"))):
                if on:
                    c = [self.t(_arr(getattr(a, w), (3, a.count))) for w in names[:3 if lor else 2]]
                    self.ade.append((half, lin, c, torch.zeros_like(c[0]), torch.zeros_like(c[0]) if lor else None))
        self.exc = [self._exc("volt"), self._exc("curr")]
        self.sig = [_arr(d.signal_volt, (d.signal_length,)), _arr(d.signal_curr, (d.signal_length,))]
        self.mur = []
        for k in range(d.num_mur):
            m = d.mur[k]
            c = [self.t(_arr(getattr(m, w), (m.n_p, m.n_pp))) for w in ("coef_p", "coef_pp")]
            self.mur.append((m.ny, m.line, m.shift, c, m.start_ts))
        self.rlc = None
        if d.rlc and d.rlc[0].count:
            r = d.rlc[0]
            pos = [_arr(r.pos[q], (r.count,), np.int64) for q in range(3)]
            lin = ((_arr(r.dir, (r.count,), np.int64) * N[0] + pos[0]) * N[1] + pos[1]) * N[2] + pos[2]
            c = {w: self.t(_arr(getattr(r, w), (r.count,))) for w in
                 ("ilv", "i2v", "vv2", "vj1", "vj2", "vvd", "ib0", "b1", "b2")}
            z = torch.zeros(r.count, dtype=torch.float64, device=self.dev)
            self.rlc = [self.t(lin), c, z, [z, z], [z, z]]  # Il, Vd[n-1], Vd[n-2], J[n-1], J[n-2]
        self.ts = 0

    def t(self, a):
        return torch.from_numpy(np.ascontiguousarray(a)).to(self.dev)

    def _exc(self, w):
        d, N = self.d, self.N
        n = getattr(d, w + "_count")
        if not n:
            return None
        p = [_arr(getattr(d, w + "_index")[q], (n,), np.int64) for q in range(3)]
        lin = ((_arr(getattr(d, w + "_dir"), (n,), np.int64) * N[0] + p[0]) * N[1] + p[1]) * N[2] + p[2]
        return self.t(lin), self.t(_arr(getattr(d, w + "_amp"), (n,))), _arr(getattr(d, w + "_delay"), (n,), np.int64)

    def _excite(self, half, F):
        if self.exc[half] is None:
            return
        lin, amp, delay = self.exc[half]
        p = self.d.signal_period_ts or self.ts + 1
        k = np.maximum(self.ts - delay, 0) % p
        k = np.where(k < self.d.signal_length, k, 0)
        F.view(-1).index_add_(0, lin, amp * self.t(self.sig[half][k]))

    def _ade_pre(self, half, F):
        for h, lin, c, A, L in self.ade:
            if h == half:
                f = F.view(3, -1)[:, lin]
                if L is not None:
                    L += c[2] * A
                    f = f - L
                A.mul_(c[0]).add_(c[1] * f)

    def _ade_apply(self, half, F):
        for h, lin, c, A, L in self.ade:
            if h == half:
                F.view(3, -1).index_add_(1, lin, -A)

    def _mur(self, stage):
        V = self.V
        for ny, line, shift, c, start in self.mur if stage < 2 else self.mur[::-1]:
            if self.ts < start:
                continue
            for q in range(2):
                f = V[(ny + 1 + q) % 3].movedim(ny, 0)  # the face's axes in (nP, nPP) order below
                a, b = f[line], f[shift]
                if ny == 1:
                    a, b = a.T, b.T
                key = (ny, line, q)
                if stage == 0:
                    self.buf[key] = b - c[q] * a
                elif stage == 1:
                    self.buf[key] = self.buf[key] + c[q] * b
                else:
                    a.copy_(self.buf[key])

    @staticmethod
    def _down(a, ax):
        return torch.cat([a.narrow(ax, 0, 1), a.narrow(ax, 0, a.shape[ax] - 1)], ax)

    def _half(self, half):
        V, I = self.V, self.I
        F = I if half else V
        self._ade_pre(half, F)
        held = []
        for sl, c, fl in self.slabs:
            held.append(c[3 * half] * F[sl] - c[3 * half + 1] * fl[half])
            F[sl] = fl[half]
        if half == 0:
            for n in range(3):
                p, q = (n + 1) % 3, (n + 2) % 3
                curl = I[q] - self._down(I[q], p) - I[p] + self._down(I[p], q)
                V[n].mul_(self.vv[n]).add_(self.vi[n] * curl)
        else:
            m = (slice(None, -1),) * 3
            for n in range(3):
                p, q = (n + 1) % 3, (n + 2) % 3

                def up(a, ax):
                    s = [slice(None, -1)] * 3
                    s[ax] = slice(1, None)
                    return a[tuple(s)]

                curl = V[q][m] - up(V[q], p) - V[p][m] + up(V[p], q)
                I[n][m] = I[n][m] * self.ii[n][m] + self.iv[n][m] * curl
        for (sl, c, fl), h in zip(self.slabs, held):
            fl[half] = F[sl].clone()
            F[sl] = h + c[3 * half + 2] * fl[half]

    def step(self):
        self.buf = {}
        self._voltages()
        self._half(1)
        self._ade_apply(1, self.I)
        self._excite(1, self.I)
        self.ts += 1

    def _voltages(self):
        V = self.V
        self._mur(0)
        if self.rlc:
            lin, c, il, vd, j = self.rlc
            il = self.rlc[2] = il + c["i2v"] * c["ilv"] * vd[0]
        self._half(0)
        self._mur(1)
        if self.rlc:
            f = V.view(-1)
            new = c["vvd"] * (f[lin] - il + c["vv2"] * vd[1] + c["vj1"] * j[0] + c["vj2"] * j[1])
            jn = c["ib0"] * (new - vd[1]) - c["b1"] * c["ib0"] * j[0] - c["b2"] * c["ib0"] * j[1]
            self.rlc[3], self.rlc[4] = [new, vd[0]], [jn, j[0]]
            f[lin] = new
        self._ade_apply(0, V)
        self._mur(2)
        self._excite(0, V)

    def probes(self):
        out = []
        for p in self.op.probes:
            a, b = list(p.start), list(p.stop)
            v = torch.zeros((), dtype=torch.float64, device=self.dev)
            if p.enabled and p.type == 0:
                for n in range(3):
                    lo, hi = min(a[n], b[n]), max(a[n], b[n])
                    if lo != hi and sum(x != y for x, y in zip(a, b)) == 1:
                        i = [a[0], a[1], a[2]]
                        i[n] = slice(lo, hi)
                        v = self.V[n][tuple(i)].sum() * (1 if a[n] < b[n] else -1)
            elif p.enabled and p.type == 1:  # a loop around z, the only current probes of these cases
                assert p.norm_dir == 2
                si, so = p.start_inside, p.stop_inside
                I = self.I
                if si[1] and si[2]:
                    v = v + I[0, a[0] + 1:b[0] + 1, a[1], a[2]].sum()
                if so[0] and si[2]:
                    v = v + I[1, b[0], a[1] + 1:b[1] + 1, a[2]].sum()
                if so[0] and so[1]:
                    v = v - I[0, a[0] + 1:b[0] + 1, b[1], b[2]].sum()
                if si[0] and so[2]:
                    v = v - I[1, a[0], a[1] + 1:b[1] + 1, b[2]].sum()
            out.append(v * p.weight)
        return torch.stack(out)

    def energy(self):
        m = (slice(None),) + (slice(None, -1),) * 3
        return EPS0 * self.V[m].square().sum() + MUE0 * self.I[m].square().sum()

    def lengths(self, dual):
        out = []
        for n in range(3):
            L = np.ctypeslib.as_array(self.d.lines[n], shape=(self.N[n],)) * self.d.unit
            if dual:
                e = np.concatenate([[L[1] - L[0]], 0.5 * (L[2:] - L[:-2]), [L[-1] - L[-2]]])
            else:
                e = np.concatenate([L[1:] - L[:-1], [L[-1] - L[-2]]])
            out.append(self.t(e).reshape([-1 if q == n else 1 for q in range(3)]))
        return out

    def dump_e_cell(self):
        out = torch.zeros_like(self.V)
        for n, e in enumerate(self.lengths(False)):
            r = self.V[n] / e
            p, q = (n + 1) % 3, (n + 2) % 3

            def cut(dp, dq):
                s = [slice(None, -1)] * 3
                s[p] = slice(1, None) if dp else slice(None, -1)
                s[q] = slice(1, None) if dq else slice(None, -1)
                return r[tuple(s)]

            out[n][:-1, :-1, :-1] = (cut(0, 0) + cut(1, 0) + cut(1, 1) + cut(0, 1)) / 4
        return out

    def dump_h_node(self, step):
        out = torch.zeros_like(self.I)
        for n, e in enumerate(self.lengths(True)):
            r = self.I[n] / e
            p, q = (n + 1) % 3, (n + 2) % 3

            def cut(dp, dq):
                s = [slice(None, -1)] * 3
                s[p] = slice(0, -2) if dp else slice(1, -1)
                s[q] = slice(0, -2) if dq else slice(1, -1)
                return r[tuple(s)]

            m = [slice(None, -1)] * 3
            m[p] = m[q] = slice(1, -1)
            out[n][tuple(m)] = (cut(0, 0) + cut(1, 0) + cut(1, 1) + cut(0, 1)) / 4
        return out[:, ::step, ::step, ::step]


def _exact_run(case, seed):
    op = Operator(_scene(case, seed))
    x = _Exact(op)
    interval = op.probe_interval
    ts, vals, en, frames = [], [], [], []
    fd, fd_int, freqs = None, 0, np.zeros(0)
    if case["freqs"]:
        freqs = np.linspace(1e9, 15e9, case["freqs"])
        nyq = [int(math.floor(1.0 / f / 2.0 / op.dT)) for f in freqs]
        freqs = np.array([f for f, k in zip(freqs, nyq) if k])
        fd_int = min([int(op.nyquist)] + [k for k in nyq if k])
        fd = np.zeros((len(op.probes), len(freqs)), np.complex128)
        dual = np.array([0.5 if p.type == 1 else 0.0 for p in op.probes])
    every = case["steps"] // case["frames"] if case["frames"] else 0

    def sample():
        if x.ts % interval == 0:
            ts.append(x.ts)
            vals.append(x.probes().cpu().numpy())
            en.append(float(x.energy()))
        if fd is not None and x.ts % fd_int == 0:
            v = x.probes().cpu().numpy()
            t = (x.ts + dual) * op.dT
            fd[...] += v[:, None] * np.exp(-2j * np.pi * freqs[None, :] * t[:, None]) * 2.0 * op.dT * fd_int

    sample()
    while x.ts < case["steps"]:
        x.step()
        sample()
        if every and x.ts % every == 0 and len(frames) < 2 * case["frames"]:
            frames += [x.dump_e_cell().cpu().numpy(), x.dump_h_node(2).cpu().numpy()]
    out = dict(V=x.V.cpu().numpy(), I=x.I.cpu().numpy(), ts=np.array(ts, np.int64), values=np.array(vals),
               energy=np.array(en))
    if frames:
        out["frames"] = frames
    if fd is not None:
        out["fd"] = fd
    return out


def exact(case, seed):
    if case["kind"] == "serve":
        return None  # thousands of timesteps for every job: minutes in 64 bits
    if case["kind"] == "batch":
        return [list(_exact_run(d, seed + 97 * k).values()) for k, d in enumerate(_job_cases(case))]
    return _exact_run(case, seed)
