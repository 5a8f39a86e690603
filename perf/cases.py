"""The solver's work as its users call it: whole runs, the per-stage driver loop,
states streamed through a case, and many resident cases at once.

Every case is a bump channel of the shapes `orion_b200.cases` and
`orion_b200.serving` build.  `prepare` makes what a program holds before it
steps (the device-resident case, its host buffers), `run` is one job on it from
the seeded initial flow to the results, and `exact` is the same job in plain
torch arithmetic in 64 bits.

The mixed path keeps its fluxes and increments in FP32, so its jobs end in the
solution output (the FP32 fields the reference writes); the plain path's jobs
return the FP64 residual history or state as well.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from orion_b200 import serving  # before the CUDA context: it asks for 32 hardware queues
from orion_b200 import _lib, cases, solver

NG = 3
OPEN = {"imin": cases.BC_FREESTREAM, "imax": cases.BC_EXTRAPOLATION, "kmax": cases.BC_EXTRAPOLATION}


def _case(name, kind, dims, split=(1, 1, 1), precision="plain", steps=4, uneven=0, moo=0.5, reynolds=1.0e3,
          height=0.05, nvis=1, open_ends=False, twall=0.0, attack=0.0):
    return {"name": name, "kind": kind, "ni": dims[0], "nj": dims[1], "nk": dims[2], "si": split[0], "sj": split[1],
            "sk": split[2], "precision": precision, "steps": steps, "uneven": uneven, "moo": moo,
            "reynolds": reynolds, "height": height, "nvis": nvis, "open_ends": open_ends, "twall": twall,
            "attack": attack}


def listed():
    return [
        # the smallest grid of the request mix, one block: pure launch and chain latency
        _case("run_33x33x33_plain", "run", (33, 33, 33), steps=4),
        # configuration 0 (one block, converging), both precisions; the mixed job is a solution run, the plain
        # one the reference driver's own loop of per-stage calls with the time step and residual read every step
        _case("run_97x49x33_mixed", "run", (97, 49, 33), precision="mixed", steps=8),
        _case("driver_97x49x33_plain", "driver", (97, 49, 33), steps=4),
        # odd sizes, uneven 1-D split, Euler, through-flow ends (freestream, extrapolation), angle of attack
        _case("euler_111x53x47_open", "run", (111, 53, 47), split=(3, 1, 1), steps=4, uneven=5, moo=0.7, nvis=0,
              open_ends=True, attack=3.0),
        # configuration 1 (8 even blocks): states streamed in and out of the case every step, and a mixed run
        _case("stream_193x97x65_plain", "stream", (193, 97, 65), split=(2, 2, 2), steps=1),
        _case("run_193x97x65_mixed", "run", (193, 97, 65), split=(2, 2, 2), precision="mixed", steps=4),
        # configuration 2 (27 uneven blocks)
        _case("run_289x161x65_plain", "run", (289, 161, 65), split=(3, 3, 3), steps=2, uneven=2, moo=0.7,
              reynolds=1.0e4),
        _case("run_289x161x65_mixed", "run", (289, 161, 65), split=(3, 3, 3), precision="mixed", steps=4, uneven=2,
              moo=0.7, reynolds=1.0e4),
        # configuration 3 (64 uneven blocks, transonic): the headline benchmark, both precisions
        _case("run_385x257x129_mixed", "run", (385, 257, 129), split=(4, 4, 4), precision="mixed", steps=4, uneven=3,
              moo=0.8, reynolds=1.0e5, height=0.08),
        _case("run_385x257x129_plain", "run", (385, 257, 129), split=(4, 4, 4), steps=2, uneven=3, moo=0.8,
              reynolds=1.0e5, height=0.08),
        # the request mix resident at once: in one group, and each case on a stream of its own
        {"name": "group_8_requests_mixed", "kind": "group", "requests": 8, "mix": 4, "precision": "mixed", "steps": 4},
        {"name": "streams_12_requests_mixed", "kind": "streams", "requests": 12, "mix": 7, "precision": "mixed",
         "steps": 4},
    ]


def draw(rng):
    kind = rng.choice(("run", "run", "run", "run", "driver", "stream", "group", "streams"))
    precision = rng.choice(("plain", "mixed"))
    if kind in ("group", "streams"):
        return {"kind": kind, "requests": rng.randint(2, 8), "mix": rng.randint(0, 1 << 20), "precision": precision,
                "steps": rng.randint(1, 3)}
    log = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))  # noqa: E731
    while True:
        dims = (log(25, 385), log(17, 257), log(13, 129))
        if dims[0] * dims[1] * dims[2] <= 4.0e6:
            break
    split = tuple(rng.randint(1, max(1, min(4, (n - 1) // 24))) for n in dims)
    nvis = rng.choice((1, 1, 1, 0))
    open_ends = rng.random() < 0.25
    c = _case("", kind, dims, split, precision, rng.randint(1, 2) if kind != "stream" else 1,
              rng.randint(1, 1 << 20) if rng.random() < 0.7 else 0, round(rng.uniform(0.2, 0.85), 3),
              round(10.0 ** rng.uniform(3.0, 5.0), 1), round(rng.uniform(0.02, 0.08), 4), nvis, open_ends,
              300.0 if rng.random() < 0.2 else 0.0, rng.choice((0.0, 0.0, 2.0)))
    if kind != "run":
        c["precision"] = "plain"  # these hand back the FP64 state
    del c["name"]
    return c


def _bump(case, seed):
    return cases.bump_case("perf", case["ni"], case["nj"], case["nk"], height=case["height"],
                           split=(case["si"], case["sj"], case["sk"]), uneven_seed=case["uneven"] or None,
                           moo=case["moo"], reynolds=case["reynolds"], noise_seed=seed, nvis=case["nvis"],
                           physical=OPEN if case["open_ends"] else None, twall=case["twall"], attack=case["attack"])


def _members(case, seed):
    reqs = serving.c4_requests(case["requests"], seed=case["mix"])
    built = [r.build_case() for r in reqs]
    for i, b in enumerate(built):
        b.noise_seed = seed * 1009 + i
    return built


def _cases_of(case, seed):
    return _members(case, seed) if case["kind"] in ("group", "streams") else [_bump(case, seed)]


class _Fields:
    """Pinned host memory for one case's solution output: 7 float fields of every block."""

    def __init__(self, fs):
        self.sizes = [7 * b.npoints for b in fs.case.blocks]
        self.buf = torch.empty(sum(self.sizes), dtype=torch.float32, pin_memory=True)

    def fetch(self, fs):
        at = self.buf.data_ptr()
        for b, n in enumerate(self.sizes):
            _lib.check(_lib.load().orion_case_pack_output(fs.handle, b, at))
            at += 4 * n
        return self.buf


def prepare(case, seed):
    prec = _lib.PREC_FP64 if case["precision"] == "plain" else _lib.PREC_MIXED
    built = _cases_of(case, seed)
    sets = [solver.FlowFieldSet(c, precision=prec) for c in built]
    state = {"case": case, "sets": sets, "group": None}
    if case["kind"] == "stream":
        prim = [torch.from_numpy(p) for p in _initial(built[0])]
        state["put"] = [p.pin_memory() for p in prim]
        state["got"] = [torch.empty_like(p).pin_memory() for p in prim]
    elif case["kind"] != "driver":
        state["fields"] = [_Fields(fs) for fs in sets]
    if case["kind"] == "group":
        state["group"] = solver.CaseGroup(sets)
    return state


def _init(fs):
    _lib.check(_lib.load().orion_case_init_flow(fs.handle, C.c_uint64(fs.case.noise_seed),
                                                C.c_double(fs.case.noise_amp)))


def _driver(fs, steps):
    halo, stats = solver.HaloExchanger(), []
    for _ in range(steps):
        halo.exchange_bc(None, fs)
        solver.apply_physical_bc(None, fs)
        solver.StateUpdater.update_flow_states(fs)
        solver.TimeIntegrator.calculate_time_step(fs)
        solver.FluxComputer.compute_viscous_rhs(fs)
        if fs.params.nvis == 1:
            halo.average_interface_residuals(None, fs)
        solver.InviscidFluxComputer.compute_inviscid_rhs(fs)
        halo.average_interface_residuals(None, fs)
        solver.StateUpdater.update_solution(fs)
        r = solver.ResidualMonitor.compute(fs)
        stats.append((r.rms_residual, r.max_residual, *r.max_loc, r.phydtime))
    return np.array(stats)


def run(state):
    case, sets, kind = state["case"], state["sets"], state["case"]["kind"]
    steps = case["steps"]
    if kind == "stream":
        fs = sets[0]
        fs.poll()
        for b, p in enumerate(state["put"]):
            fs.io_put(b, p)
        fs.io_step(steps)
        for b, p in enumerate(state["got"]):
            fs.io_get(b, p)
        return state["got"]
    for fs in sets:
        _init(fs)
    if kind == "driver":
        hist = _driver(sets[0], steps)
        return {"hist": hist, "prim": [sets[0].download(b, "prim") for b in range(len(sets[0].case.blocks))]}
    if kind == "run":
        if case["precision"] == "plain":
            return {"hist": sets[0].step(steps), "fields": state["fields"][0].fetch(sets[0])}
        sets[0].step_async(steps)
        return {"fields": state["fields"][0].fetch(sets[0])}
    if kind == "group":
        state["group"].submit(steps)
        state["group"].sync()
    else:
        for fs in sets:
            fs.submit(steps)
        for fs in sets:
            fs.sync()
    for fs in sets:
        fs.poll()
    return {"fields": [f.fetch(fs) for f, fs in zip(state["fields"], sets)]}


#: Arithmetic operations per point and step, counted from the formulas: inviscid 3 x (5 x 2 WCNS states of 55, a Roe
#: flux of 180, metric and difference 60), viscous 3 x 260 and its 12 node derivatives, sweeps 18 neighbour terms of
#: 65, derived state, time step and update 180.
FLOPS_EULER, FLOPS_VISCOUS = 3 * (550 + 180 + 60) + 18 * 65 + 180, 3 * 260 + 12 * 8


def work(case):
    if case["kind"] in ("group", "streams"):
        pts = sum(r.npoints for r in serving.c4_requests(case["requests"], seed=case["mix"]))
        nvis = 1
    else:
        pts, nvis = case["ni"] * case["nj"] * case["nk"], case["nvis"]
    # per step: the primitive state in and out, the metrics and the Jacobian in; then the results once
    step = (2 * 6 + 9 + 1) * 8
    out = 28 if case["kind"] not in ("stream", "driver") else 48
    flops = FLOPS_EULER + (FLOPS_VISCOUS if nvis == 1 else 0)
    return {"bytes": pts * (case["steps"] * step + out), "flops": pts * case["steps"] * flops}


# --------------------------------------------------------------------------- the same jobs in plain 64-bit arithmetic
def _noise(seed, first, count):
    """Draws first+1 .. first+count of splitmix64(seed), in [0, 1)."""
    with np.errstate(over="ignore"):
        z = np.uint64(seed) + np.arange(first + 1, first + count + 1, dtype=np.uint64) * np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        z = z ^ (z >> np.uint64(31))
    return (z >> np.uint64(11)).astype(np.float64) / 2.0 ** 53


def _initial(c):
    """Padded primitive state (6, nz, ny, nx) of every block: freestream, seeded noise on rho and u."""
    p, first, out = c.params, 0, []
    for b in c.blocks:
        shape = tuple(n + 2 * NG for n in (b.kdim, b.jdim, b.idim))
        n = int(np.prod(shape))
        r = _noise(c.noise_seed, 2 * first, 2 * n).reshape(n, 2)
        first += n
        prim = np.empty((6,) + shape)
        prim[0] = p.roo * (1.0 + c.noise_amp * (2.0 * r[:, 0].reshape(shape) - 1.0))
        prim[1] = p.uoo * (1.0 + c.noise_amp * (2.0 * r[:, 1].reshape(shape) - 1.0))
        prim[2], prim[3], prim[4] = p.voo, p.woo, p.poo
        prim[5] = p.moo * p.moo * (p.gamma * prim[4] / prim[0]) if p.nvis == 1 else p.too
        out.append(prim)
    return out


def _face_values(q, n):
    """Line values q[0..n) (first axis) to faces 0..n, one-sided at the ends."""
    h = torch.empty((n + 1,) + q.shape[1:], dtype=q.dtype, device=q.device)
    h[2:n - 1] = (9 * (q[1:n - 2] + q[2:n - 1]) - (q[3:n] + q[0:n - 3])) / 16
    for s, e in ((1, lambda t: q[t]), (-1, lambda t: q[n - 1 - t])):
        f = (lambda t: t) if s == 1 else (lambda t: n - t)
        h[f(0)] = (35 * e(0) - 35 * e(1) + 21 * e(2) - 5 * e(3)) / 16
        h[f(1)] = (5 * e(0) + 15 * e(1) - 5 * e(2) + e(3)) / 16
    return h


def _difference(f, n):
    """Sixth-order difference of face values 0..n at points 0..n-1, one-sided at the ends."""
    d = torch.empty((n,) + f.shape[1:], dtype=f.dtype, device=f.device)
    d[2:n - 2] = (2250 * (f[3:n - 1] - f[2:n - 2]) - 125 * (f[4:n] - f[1:n - 3]) + 9 * (f[5:n + 1] - f[0:n - 4])) / 1920
    d[0] = (-23 * f[0] + 21 * f[1] + 3 * f[2] - f[3]) / 24
    d[1] = (f[0] - 27 * f[1] + 27 * f[2] - f[3]) / 24
    d[n - 1] = -(-23 * f[n] + 21 * f[n - 1] + 3 * f[n - 2] - f[n - 3]) / 24
    d[n - 2] = -(f[n] - 27 * f[n - 1] + 27 * f[n - 2] - f[n - 3]) / 24
    return d


def _along(a, d):
    """Moves grid direction d (0 = i) of an array (..., k, j, i) to the front."""
    return torch.movedim(a, a.ndim - 1 - d, 0)


def _back(a, d):
    return torch.movedim(a, 0, a.ndim - 1 - d)


def _metrics(b, dev):
    """Metrics (9, k, j, i) in the conservative form, and the Jacobian."""
    x = torch.stack([torch.from_numpy(np.asarray(v, dtype=np.float64)) for v in (b.x, b.y, b.z)]).to(dev)

    def der(a, d):
        n = a.shape[a.ndim - 1 - d]
        return _back(_difference(_face_values(_along(a, d), n), n), d)

    g = [der(x, d) for d in range(3)]  # g[d][c] = d x_c / d xi_d
    met = []
    for d in range(3):
        e, f = (d + 1) % 3, (d + 2) % 3
        for c in range(3):
            a, q = (c + 1) % 3, (c + 2) % 3
            # d/df (x_a,e x_q) - d/de (x_a,f x_q)
            met.append(der(g[e][a] * x[q], f) - der(g[f][a] * x[q], e))
    met = torch.stack(met)
    vol = g[0][0] * met[0] + g[1][0] * met[3] + g[2][0] * met[6]
    return met, torch.where(vol < 1e-15, torch.full_like(vol, 1e-15), vol)


class _Block:
    def __init__(self, b, prim, p, dev):
        self.b, self.p = b, p
        self.n = (b.idim, b.jdim, b.kdim)
        self.prim = torch.from_numpy(prim).to(dev)
        met, vol = _metrics(b, dev)
        pad = (NG,) * 6
        self.met = torch.nn.functional.pad(met, pad)
        self.vol = torch.nn.functional.pad(vol, pad)
        self.mu = torch.zeros_like(self.vol)
        self.mask = torch.zeros(self.vol.shape, dtype=torch.bool, device=dev)
        for r in b.regions:
            if r.bctype > 0:
                self.mask[self._window(r)] = True

    def inner(self, a):
        return a[..., NG:-NG, NG:-NG, NG:-NG]

    def _window(self, r):
        return tuple(slice(r.s_st[d] - 1 + NG, r.s_ed[d] + NG) for d in (2, 1, 0))

    def layers(self, a, r, at):
        """Plane `at` of array a off a face region: 0 the face, > 0 ghosts, < 0 inside."""
        d = next(m for m in range(3) if r.s_st[m] == r.s_ed[m])
        hi = r.s_st[d] != 1
        face = r.s_st[d] - 1 + NG
        w = list(self._window(r))
        w[2 - d] = face + at if hi else face - at
        return a[(Ellipsis,) + tuple(w)]

    def boundary(self, r):
        p, q = self.p, self.prim
        d = next(m for m in range(3) if r.s_st[m] == r.s_ed[m])
        at = lambda k: self.layers(q, r, k)  # noqa: E731
        m = self.layers(self.met[3 * d:3 * d + 3], r, 0)
        nrm = m / torch.clamp((m * m).sum(0).sqrt(), min=1e-30)
        mean = False
        if r.bctype == cases.BC_WALL and p.nvis == 1:
            a, b = at(-1).clone(), at(-2).clone()
            pw = (4 * a[4] - b[4]) / 3
            pw = torch.where(pw < 1e-6, a[4], pw)
            if p.twall > 1e-6:
                tw = torch.full_like(pw, p.twall / p.tref)
            else:
                tw = (4 * a[5] - b[5]) / 3
                tw = torch.where(tw < 1e-6, a[5], tw)
            k = p.moo * p.moo * p.gamma
            for l in (1, 2, 3):
                g, i = at(l), at(-l)
                g[1:4] = -i[1:4]
                g[4] = i[4]
                g[5] = 2 * tw - i[5] if p.twall > 1e-6 else i[5]
                rho = k * g[4] / torch.where(g[5] < 1e-6, torch.ones_like(tw), g[5])
                g[0] = -rho if l == 3 else rho
            f = at(0)
            f[0], f[1:4], f[4], f[5] = k * pw / tw, 0.0, pw, tw
        elif r.bctype in (cases.BC_WALL, cases.BC_SYMMETRY):
            if r.bctype == cases.BC_SYMMETRY:  # one normal for the face: its middle point's
                lo = [s - 1 for s in r.s_st]
                mid = [(s - 1 + e - 1) // 2 if s != e else 0 for s, e in zip(r.s_st, r.s_ed)]
                at2 = [m_ - l_ for c, (m_, l_) in enumerate(zip(mid, lo)) if c != d][::-1]
                nrm = nrm[:, at2[0], at2[1]][:, None, None]
            for l in (1, 2, 3):
                g, i = at(l), at(-l).clone()
                vn = (i[1:4] * nrm).sum(0)
                g[0] = -i[0] if (r.bctype == cases.BC_WALL and l == 3) else i[0]
                g[1:4] = i[1:4] - 2 * vn * nrm
                g[4:6] = i[4:6]
            mean = p.method == 1
        elif r.bctype == cases.BC_FARFIELD:
            if r.s_st[d] == 1:
                nrm = -nrm
            ga, g1 = p.gamma, p.gamma - 1
            i = at(-1).clone()
            ci, cf = (ga * i[4] / i[0]).sqrt(), math.sqrt(ga * p.poo / p.roo)
            ent_i, ent_f = i[4] / i[0] ** ga, p.poo / p.roo ** ga
            free = torch.tensor([p.uoo, p.voo, p.woo], dtype=q.dtype, device=q.device)[:, None, None]
            vi, vf = (i[1:4] * nrm).sum(0), (free * nrm).sum(0)
            mach = (i[1:4] ** 2).sum(0).sqrt() / ci
            rp, rm = vi + 2 * ci / g1, vf - 2 * cf / g1
            vb, cb = 0.5 * (rp + rm), 0.25 * g1 * (rp - rm)
            outflow = vb > 0
            ent = torch.where(outflow, ent_i, torch.full_like(ent_i, ent_f))
            ref, vr = torch.where(outflow, i[1:4], free), torch.where(outflow, vi, vf)
            rb = (cb * cb / (ga * ent)) ** (1 / g1)
            s = torch.empty_like(i)
            sub = mach < 1
            s[0] = torch.where(sub, rb, torch.where(vi > 0, i[0], torch.full_like(rb, p.roo)))
            s[4] = torch.where(sub, ent * rb ** ga, torch.where(vi > 0, i[4], torch.full_like(rb, p.poo)))
            s[1:4] = torch.where(sub, ref + (vb - vr) * nrm, torch.where(vi > 0, i[1:4], free))
            s[5] = mach * mach * ga * s[4] / s[0]
            for l in (1, 2, 3):
                g = at(l)
                g[:] = s
                if l == 3:
                    g[0] = -s[0]
        elif r.bctype == cases.BC_FREESTREAM:
            s = torch.tensor([p.roo, p.uoo, p.voo, p.woo, p.poo, p.too], dtype=q.dtype, device=q.device)
            for l in (1, 2, 3):
                at(l)[:] = s[:, None, None]
        elif r.bctype == cases.BC_EXTRAPOLATION:
            s = at(-1).clone()
            for l in (1, 2, 3):
                at(l)[:] = s
        if mean:
            at(0)[:] = 0.5 * (at(1) + at(-1))

    def derived(self):
        p, q = self.p, self.prim
        box = torch.zeros(self.vol.shape, dtype=torch.int8, device=q.device)
        for d in range(3):
            v = _along(box, d)
            v[NG:-NG] += 1
        rho = torch.where(box == 2, q[0].abs(), q[0])
        a2 = p.gamma * q[4] / rho
        self.c = torch.where(box >= 2, a2.abs().sqrt(), torch.zeros_like(a2))
        if p.nvis == 1:
            q[5] = torch.where(box >= 2, p.moo * p.moo * a2, q[5])
            t = torch.clamp(q[5], min=1e-6)
            self.mu = t * t.sqrt() * (1 + p.visc) / (t + p.visc)
        r, v = self.inner(q), self.inner(self.vol)
        met, c, mu = self.inner(self.met), self.inner(self.c), self.inner(self.mu)
        tot = 0
        for d in range(3):
            m = met[3 * d:3 * d + 3]
            g2 = (m * m).sum(0)
            tot = tot + (r[1:4] * m).sum(0).abs() + c * g2.sqrt()
            if p.nvis == 1:
                tot = tot + 2 * mu / (p.reynolds * r[0] * v + 1e-30) * g2 * p.csrv
        self.dt = p.cfl / (tot + 1e-30) / v
        self.dq = torch.zeros((5,) + v.shape, dtype=q.dtype, device=q.device)

    def _lines(self, a, d):
        """A padded array with direction d in front and the other two directions' ghosts cut off."""
        cut = [slice(NG, -NG)] * 3
        cut[2 - d] = slice(None)
        return _along(a[(Ellipsis,) + tuple(cut)], d)

    def viscous(self):
        p, n3 = self.p, self.n
        var = self.prim[[1, 2, 3, 5]]
        node = []
        for d in range(3):
            n, x = n3[d], self._lines(var, d)
            rho = self._lines(self.prim[0], d)
            y = (8 * (x[4:n + 4] - x[2:n + 2]) - (x[5:n + 5] - x[1:n + 1])) / 12
            for flag, e, s, k in ((rho[0] < 0, lambda t: x[3 + t], 1, lambda t: t),
                                  (rho[n + 5] < 0, lambda t: x[n + 2 - t], -1, lambda t: n - 1 - t)):
                y[k(0)] = torch.where(flag, s * (-11 * e(0) + 18 * e(1) - 9 * e(2) + 2 * e(3)) / 6, y[k(0)])
                y[k(1)] = torch.where(flag, s * (-3 * e(0) - 10 * e(1) + 18 * e(2) - 6 * e(3) + e(4)) / 12, y[k(1)])
            node.append(_back(y, d))
        for d in range(3):
            n, x = n3[d], self._lines(var, d)
            rho = self._lines(self.prim[0], d)
            half = lambda a: (9 * (a[2:n + 3] + a[3:n + 4]) - (a[4:n + 5] + a[1:n + 2])) / 16  # noqa: E731
            u, du = half(x), (27 * (x[3:n + 4] - x[2:n + 3]) - (x[4:n + 5] - x[1:n + 2])) / 24
            for flag, e, s, k in ((rho[0] < 0, lambda t: x[3 + t], 1, lambda t: t),
                                  (rho[n + 5] < 0, lambda t: x[n + 2 - t], -1, lambda t: n - t)):
                u[k(0)] = torch.where(flag, (35 * e(0) - 35 * e(1) + 21 * e(2) - 5 * e(3)) / 16, u[k(0)])
                u[k(1)] = torch.where(flag, (5 * e(0) + 15 * e(1) - 5 * e(2) + e(3)) / 16, u[k(1)])
                du[k(0)] = torch.where(flag, s * (-71 * e(0) + 141 * e(1) - 93 * e(2) + 23 * e(3)) / 24, du[k(0)])
                du[k(1)] = torch.where(flag, s * (-22 * e(0) + 17 * e(1) + 9 * e(2) - 5 * e(3) + e(4)) / 24, du[k(1)])
            mu, vol, met = (half(self._lines(a, d)) for a in (self.mu, self.vol, self.met))
            der = []
            for m in range(3):
                if m == d:
                    der.append(du)
                else:  # the node derivatives' end values stand in for the ghosts
                    y = _along(node[m], d)
                    y = torch.cat([y[:1]] * 3 + [y] + [y[-1:]] * 3)
                    der.append(half(y))
            g = [[(met[:, c] * der[0][:, v] + met[:, c + 3] * der[1][:, v] + met[:, c + 6] * der[2][:, v]) / vol
                  for c in range(3)] for v in range(4)]
            div = g[0][0] + g[1][1] + g[2][2]
            nrm = [met[:, 3 * d + c] for c in range(3)]
            f = []
            for a in range(3):
                t = 0
                for c in range(3):
                    tau = mu * (g[a][c] + g[c][a])
                    if a == c:
                        tau = tau - mu * (2.0 / 3.0) * div
                    t = t + tau * nrm[c]
                f.append(t)
            k = mu / ((p.gamma - 1) * p.moo * p.moo) / p.prl
            f.append(u[:, 0] * f[0] + u[:, 1] * f[1] + u[:, 2] * f[2] +
                     k * (g[3][0] * nrm[0] + g[3][1] * nrm[1] + g[3][2] * nrm[2]))
            self.dq[1:] -= _back(_difference(torch.stack(f, 1), n), d) / p.reynolds

    def inviscid(self):
        for d in range(3):
            n = self.n[d]
            x = self._lines(self.prim[:5], d)  # (n + 6, 5, a, b)
            lo, hi = x[0, 0] < 1e-20, x[n + 5, 0] < 1e-20
            kx = _face_values(self._lines(self.met[3 * d:3 * d + 3], d)[NG:NG + n], n)
            a = [x[m:m + n + 1] for m in range(6)]
            left, right = _wcns(a[0], a[1], a[2], a[3], a[4]), _wcns(a[5], a[4], a[3], a[2], a[1])
            first, last = [x[3 + t] for t in range(4)], [x[n + 2 - t] for t in range(4)]
            wl, wr = left.clone(), right.clone()
            for flag, e, k, inner in ((lo, first, lambda t: t, wl), (hi, last, lambda t: n - t, wr)):
                e0 = (35 * e[0] - 35 * e[1] + 21 * e[2] - 5 * e[3]) / 16
                e1 = (5 * e[0] + 15 * e[1] - 5 * e[2] + e[3]) / 16
                e2 = (-e[0] + 9 * e[1] + 9 * e[2] - e[3]) / 16
                for s in (wl, wr):
                    s[k(0)] = torch.where(flag, e0, s[k(0)])
                    s[k(1)] = torch.where(flag, e1, s[k(1)])
                inner[k(2)] = torch.where(flag, e2, inner[k(2)])

            def flux(face, l, r):
                """The Roe flux at faces `face` (a slice or index), with the positivity fallback."""
                idx = torch.arange(n + 1, device=x.device)[face]
                l = torch.where(((l.select(-3, 0) <= 1e-6) | (l.select(-3, 4) <= 1e-6)).unsqueeze(-3),
                                x[torch.clamp(idx - 1, min=0) + 2], l)
                r = torch.where(((r.select(-3, 0) <= 1e-6) | (r.select(-3, 4) <= 1e-6)).unsqueeze(-3),
                                x[torch.clamp(idx, max=n - 1) + 3], r)
                return _roe(l, r, kx[face], self.p.gamma)

            f = _difference(flux(slice(0, n + 1), wl, wr), n)
            for flag, e, k, s in ((lo, first, lambda t: t, 1), (hi, last, lambda t: n - t, -1)):
                pt = (lambda t: t) if s == 1 else (lambda t: n - 1 - t)
                q3, q4, q5, q6 = e
                one = lambda t, v: flux(k(t), v, v)  # noqa: E731
                # `near` is the side of the flagged end: the left state at the low end
                two = (lambda t, near, far: flux(k(t), near, far)) if s == 1 else \
                      (lambda t, near, far: flux(k(t), far, near))
                other = right if s == 1 else left
                r0 = -23 * one(0, (3 * q3 - q4) / 2) + 21 * one(1, (19 * q3 + 25 * q4 - 2 * q5) / 42) + \
                    3 * one(2, (4 * q3 + 3 * q4 + 9 * q5 + 2 * q6) / 18) - one(3, (-2 * q3 + 3 * q4 + 3 * q5 + 2 * q6) / 6)
                b1, b3, b4 = (3 * q3 + 6 * q4 - q5) / 8, (-q4 + 6 * q5 + 3 * q6) / 8, (q4 + 2 * q5 + 5 * q6) / 8
                r1 = -22 * one(1, b1) + 17 * two(2, (-30 * q3 + 145 * q4 + 29 * q5 - 8 * q6) / 136,
                                                 (2 * q3 + 49 * q4 + 125 * q5 - 40 * q6) / 136) + \
                    9 * one(3, b3) - 5 * one(4, b4) + one(5, (q4 + q5 + 6 * q6) / 8)
                r2 = two(1, b1, (5 * q3 + 15 * q4 - 5 * q5 + q6) / 16) - \
                    27 * two(2, (-29 * q3 + 170 * q4 + 63 * q5 + 12 * q6) / 216, other[k(2)]) + \
                    27 * two(3, b3, other[k(3)]) - two(4, b4, other[k(4)])
                for t, v in enumerate((r0, r1, r2)):
                    f[pt(t)] = torch.where(flag, s * v / 24, f[pt(t)])
            self.dq += _back(f, d)


def _wcns(a, b, c, d, e):
    """The WCNS-E-5 state on the d side of point c."""
    s = (a - 2 * b + c, b - 2 * c + d, c - 2 * d + e)
    g = (0.5 * (a - 4 * b + 3 * c), 0.5 * (d - b), 0.5 * (-3 * c + 4 * d - e))
    w = [k / (1e-6 + gi * gi + si * si) ** 2 for k, gi, si in zip((1 / 16, 10 / 16, 5 / 16), g, s)]
    return c + 0.125 * sum(wi * (si + 4 * gi) for wi, si, gi in zip(w, s, g)) / (w[0] + w[1] + w[2])


def _physical(q, ga, k):
    r, u, v, w, p = (q.select(-3, m) for m in range(5))
    kx, ky, kz = (k.select(-3, m) for m in range(3))
    vn = u * kx + v * ky + w * kz
    h = (p / (ga - 1) + 0.5 * r * (u * u + v * v + w * w) + p) / r
    return torch.stack([r * vn, r * u * vn + p * kx, r * v * vn + p * ky, r * w * vn + p * kz, r * h * vn], -3)


def _roe(l, r, k, ga):
    kx, ky, kz = (k.select(-3, m) for m in range(3))
    ql, qr = [l.select(-3, m) for m in range(5)], [r.select(-3, m) for m in range(5)]
    h = [ga / (ga - 1) * q[4] / q[0] + 0.5 * (q[1] * q[1] + q[2] * q[2] + q[3] * q[3]) for q in (ql, qr)]
    sl, sr = ql[0].sqrt(), qr[0].sqrt()
    mean = lambda a, b: (sl * a + sr * b) / (sl + sr)  # noqa: E731
    rho, hm = sl * sr, mean(*h)
    vel = [mean(ql[m], qr[m]) for m in (1, 2, 3)]
    v2 = vel[0] ** 2 + vel[1] ** 2 + vel[2] ** 2
    c2 = (hm - 0.5 * v2) * (ga - 1)
    c2 = torch.where(c2 <= 0, torch.full_like(c2, 1e-6), c2)
    c, gm = c2.sqrt(), torch.clamp((kx * kx + ky * ky + kz * kz).sqrt(), min=1e-30)
    un, nrm, cg = vel[0] * kx + vel[1] * ky + vel[2] * kz, (kx / gm, ky / gm, kz / gm), c * gm
    delta = 0.1 * cg
    fix = lambda a: torch.where(a.abs() < delta, (a * a + delta * delta).sqrt(), a.abs())  # noqa: E731
    l1, l4, l5 = fix(un - cg), fix(un), fix(un + cg)
    dv = [qr[m] - ql[m] for m in (1, 2, 3)]
    drho, dp = qr[0] - ql[0], qr[4] - ql[4]
    dn = rho * (dv[0] * nrm[0] + dv[1] * nrm[1] + dv[2] * nrm[2])
    a1 = l4 * (drho - dp / c2)
    a2, a3 = 0.5 * l5 * (dp / c2 + dn / c), 0.5 * l1 * (dp / c2 - dn / c)
    a4, a5 = a1 + a2 + a3, c * (a2 - a3)
    t = [l4 * (rho * dv[m] - nrm[m] * dn) for m in range(3)]
    df = [a4] + [vel[m] * a4 + nrm[m] * a5 + t[m] for m in range(3)]
    df.append(hm * a4 + un / gm * a5 + vel[0] * t[0] + vel[1] * t[1] + vel[2] * t[2] - c2 * a1 / (ga - 1))
    return 0.5 * (_physical(l, ga, k) + _physical(r, ga, k) - torch.stack(df, -3))


class _Sweeps:
    """Every block's interior points by hyperplane i + j + k, blocks side by side."""

    def __init__(self, blocks, dev):
        plane, nbr, base = [], [], 0
        for b in blocks:
            ni, nj, nk = b.n
            k, j, i = torch.meshgrid(*(torch.arange(m, device=dev) for m in (nk, nj, ni)), indexing="ij")
            at = base + i + ni * (j + nj * k)
            plane.append((i + j + k).reshape(-1))
            one = []
            for x, m, st in ((i, ni, 1), (j, nj, ni), (k, nk, ni * nj)):
                one.append((torch.where(x > 0, at - st, -1), torch.where(x < m - 1, at + st, -1)))
            nbr.append(torch.stack([o[0].reshape(-1) for o in one] + [o[1].reshape(-1) for o in one]))
            base += ni * nj * nk
        plane = torch.cat(plane)
        self.order = torch.argsort(plane, stable=True)
        rank = torch.empty_like(self.order)
        rank[self.order] = torch.arange(base, device=dev)
        nb = torch.cat(nbr, 1)[:, self.order]
        self.there = nb >= 0
        self.nb = torch.where(self.there, rank[nb.clamp(min=0)], 0)
        count = torch.bincount(plane).tolist()
        self.off = [0]
        for m in count:
            self.off.append(self.off[-1] + m)
        self.rank = rank

    def solve(self, prim, mu, vol, met, dt, rhs, p):
        """The four sweeps' increment; arguments by point in the blocks' own order."""
        o = self.order
        q, mu, vol, met, rhs = prim[:, o], mu[o], vol[o].clamp(min=1e-30), met[:, o], rhs[:, o]
        ga, g1 = p.gamma, p.gamma - 1
        c2 = ga * q[4].clamp(min=1e-30) / q[0].clamp(min=1e-30)
        c, v2 = c2.sqrt(), q[1] ** 2 + q[2] ** 2 + q[3] ** 2
        h, af = c2 / g1 + 0.5 * v2, 0.5 * g1 * v2
        visc = 2 * mu / (abs(p.reynolds) * q[0].clamp(min=1e-30) * vol + 1e-30) if p.nvis == 1 else torch.zeros_like(c)
        tot = 1 / dt[o]
        pair = []
        for d in range(3):
            m = met[3 * d:3 * d + 3]
            g2 = (m * m).sum(0)
            tot = tot + (q[1:4] * m).sum(0).abs() + c * g2.sqrt() + visc * g2
        coed = 1 / tot
        for s in range(6):
            m = met[3 * (s % 3):3 * (s % 3) + 3]
            g2, n = (m * m).sum(0), self.nb[s]
            gm = g2.sqrt().clamp(min=1e-30)
            ct = (q[1:4, n] * m).sum(0)
            r = ct.abs() + c[n] * gm
            l1 = 0.5 * (ct + (r if s < 3 else -r))
            # the acoustic pair's mean equals l1 and its half difference is c |grad| / 2
            pair.append((l1, 0.5 * gm, ct / gm, 0.5 * visc[n] * g2, m / gm))
        dq = torch.zeros_like(rhs)

        def term(s, a, b):
            n = self.nb[s][a:b]
            l1, x2, ctn, rv, nrm = (v[..., a:b] for v in pair[s])
            x, vel = dq[:, n], q[1:4, n]
            dc = ctn * x[0] - (nrm * x[1:4]).sum(0)
            dh = af[n] * x[0] - g1 * ((vel * x[1:4]).sum(0) - x[4])
            f = l1 * x
            f[0] -= dc * x2
            f[1:4] += (nrm * dh - vel * dc) * x2
            f[4] += (ctn * dh - h[n] * dc) * x2
            return torch.where(self.there[s][a:b], f, torch.zeros_like(f)), torch.where(self.there[s][a:b], rv * x, 0 * x)

        planes = list(zip(self.off[:-1], self.off[1:]))
        for a, b in planes:
            dq[:, a:b] = (sum(sum(term(s, a, b)) for s in (0, 1, 2)) - rhs[:, a:b]) * coed[a:b]
        for a, b in planes[::-1]:
            dq[:, a:b] = dq[:, a:b] - sum(sum(term(s, a, b)) for s in (3, 4, 5)) * coed[a:b]
        for seq in (planes, planes[::-1]):
            for a, b in seq:
                t = -rhs[:, a:b]
                for s in range(6):
                    f, rv = term(s, a, b)
                    t = t + f + rv if s < 3 else t - f + rv
                dq[:, a:b] = t * coed[a:b]
        return dq[:, self.rank]


def _updated(q, dq, g1):
    r, e = q[0], q[4] / g1 + 0.5 * q[0] * (q[1] ** 2 + q[2] ** 2 + q[3] ** 2)
    cons = torch.stack([r, r * q[1], r * q[2], r * q[3], e])
    press = lambda s: g1 * (s[4] - 0.5 * (s[1] ** 2 + s[2] ** 2 + s[3] ** 2) / s[0])  # noqa: E731
    rel = ((press(cons + dq) - q[4]) / q[4]).abs()
    new = cons + dq / (1 + 2 * (rel - 0.3).clamp(min=0))
    pn = press(new)
    out = torch.stack([new[0], new[1] / new[0], new[2] / new[0], new[3] / new[0], pn])
    return torch.where(~((new[0] <= 1e-6) | (pn <= 1e-6)), out, q)


def _march(c, steps, dev):
    """`steps` steps from the initial flow: the blocks, and (steps, 8) residual statistics."""
    p = c.params
    blocks = [_Block(b, q, p, dev) for b, q in zip(c.blocks, _initial(c))]
    sweeps = _Sweeps(blocks, dev)
    flat = lambda get: torch.cat([get(b).reshape(*get(b).shape[:-3], -1) for b in blocks], -1)  # noqa: E731
    vol, met = flat(lambda b: b.inner(b.vol)), flat(lambda b: b.inner(b.met))
    mask = flat(lambda b: b.inner(b.mask))
    total, hist = vol.numel(), np.zeros((steps, 8))

    def average():
        dens = [(b.dq / b.inner(b.vol)) for b in blocks]
        full = lambda a: torch.nn.functional.pad(a, (NG,) * 6)  # noqa: E731
        packed = [full(d) for d in dens]
        for b in blocks:
            for r in b.b.regions:
                if r.bctype < 0:
                    t = blocks[r.nbt - 1]
                    other = t.layers(packed[r.nbt - 1], t.b.regions[r.ibcwin - 1], 0)
                    wide = full(b.dq)
                    mine = b.layers(wide, r, 0)
                    mine[:] = 0.5 * (other * b.layers(b.vol, r, 0) + mine)
                    b.dq = b.inner(wide).contiguous()

    for s in range(steps):
        for b in blocks:  # ghosts of an interface: the neighbour's interface plane and the two inside it
            for r in b.b.regions:
                if r.bctype < 0:
                    t = blocks[r.nbt - 1]
                    tr = t.b.regions[r.ibcwin - 1]
                    for l in (1, 2, 3):
                        b.layers(b.prim[:5], r, l)[:] = t.layers(t.prim[:5], tr, 1 - l)
        for b in blocks:
            for r in b.b.regions:
                if r.bctype > 0:
                    b.boundary(r)
            b.derived()
            if p.nvis == 1:
                b.viscous()
        if p.nvis == 1:
            average()
        for b in blocks:
            b.inviscid()
        average()
        prim, dt = flat(lambda b: b.inner(b.prim)[:5]), flat(lambda b: b.dt)
        dq = sweeps.solve(prim, flat(lambda b: b.inner(b.mu)), vol, met, dt,
                          torch.where(mask, 0.0, flat(lambda b: b.dq)), p)
        dq = torch.where(mask, 0.0, dq)
        new = _updated(prim, dq, p.gamma - 1)
        res = dq.abs() / (dt.clamp(min=1e-30) * vol.clamp(min=1e-30))
        key = int(torch.argmax(res.t().reshape(-1)))
        at = 0
        for nb, b in enumerate(blocks):
            ni, nj, nk = b.n
            b.inner(b.prim)[:5] = new[:, at:at + ni * nj * nk].reshape(5, nk, nj, ni)
            pt = key // 5 - at
            if 0 <= pt < ni * nj * nk:
                hist[s, 2:7] = nb, pt % ni + 1, pt // ni % nj + 1, pt // (ni * nj) + 1, key % 5 + 1
            at += ni * nj * nk
        hist[s, 0], hist[s, 1] = float((res * res).sum() / (5 * total)) ** 0.5, float(res.max())
        hist[s, 7] = min(1000.0, float((dt * vol).min()))
    return blocks, hist


def _output_fields(blocks, ga):
    out = []
    for b in blocks:
        r, u, v, w, p, t = b.inner(b.prim)
        mach = ((u * u + v * v + w * w) / (ga * p / r)).sqrt()
        out.append(torch.stack([r, p, t, mach, u, v, w]).reshape(-1))
    return torch.cat(out)


def exact(case, seed):
    built = _cases_of(case, seed)
    chain = sum(sum(max(sum(b.dims) for b in c.blocks) for _ in range(case["steps"])) for c in built)
    points = case["steps"] * sum(c.npoints for c in built)
    if 6e-3 * chain + 4e-7 * points > 20:  # dependent hyperplanes, and the points' arithmetic, in seconds
        return None
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    done = [_march(c, case["steps"], dev) for c in built]
    blocks, hist = done[0]
    if case["kind"] == "stream":
        return [b.prim.cpu() for b in blocks]
    if case["kind"] == "driver":
        return {"hist": hist, "prim": [b.prim.cpu() for b in blocks]}
    fields = [_output_fields(b, c.params.gamma).cpu() for (b, _), c in zip(done, built)]
    if case["kind"] == "run":
        return {"hist": hist, "fields": fields[0]} if case["precision"] == "plain" else {"fields": fields[0]}
    return {"fields": fields}
