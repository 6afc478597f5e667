"""The work this engine is measured on: what a program that simulates clump avalanches has it do.

A program holds a context (the C ABI of include/af3d.h), hands it the particle array, takes K
steps and reads the particles back; or keeps the particles on the host and takes one step a call;
or drives the step routine by routine as the reference's loop does; or asks for the gradients of
a run.  Every case is one of these calls on a flow that is moving: sheared downslope speed,
random velocities on top and spins, so that contacts load, slide and separate as they do in an
avalanche (or in a filling hopper, or in a hopper discharging through the funnel).
"""
from __future__ import annotations

import ctypes as C
import dataclasses
import math

import numpy as np
import torch

from avalancheflume3d_gb300 import (FP_EXACT, FP_FAST, FRICTION_DEV, FRICTION_HST, PARTICLE, PHASE_AVALANCHE,
                                    PHASE_FILL, Engine, lib)
from avalancheflume3d_gb300.workloads import ensemble_configs, ensemble_state, flume_2k, flume_state, funnel_524k

FIELDS = ("rr", "vv", "ww", "Rmatx", "Rmaty", "Rmatz", "rr_s")
ADJ_PARAMS = ("kappa_pp", "gamma_pp", "mu_pp", "kappa_pw", "gamma_pw", "mu_pw")


def _case(call, n, steps, layout="bed", mode="fast", friction="hst", flumes=1, length=40.0, width=4.0, tilt=30.0,
          spread=0.0, **kw):
    return {"call": call, "n": n, "steps": steps, "layout": layout, "mode": mode, "friction": friction,
            "flumes": flumes, "length": length, "width": width, "tilt": tilt, "spread": spread, **kw}


def listed():
    return [
        # the smallest run in use (a laboratory chute, a test): launches and latency count
        _case("step", 512, 200, mode="exact", name="chute512_exact"),
        # the 2,048-clump flume of the benchmark, one stretch between two snapshots
        _case("step", 2048, 500, name="flume2k_fast"),
        # an ordinary flume at an odd count, the default arithmetic, the device friction law
        _case("step", 9973, 100, mode="exact", friction="dev", name="flume9973_exact_dev"),
        # the 32,768-clump flume, fast arithmetic
        _case("step", 32768, 100, length=80.0, tilt=35.0, name="flume32k_fast"),
        # the benchmark's headline flume in either arithmetic
        _case("step", 262144, 40, length=200.0, width=20.0, tilt=35.0, name="flume262k_fast"),
        _case("step", 262144, 20, mode="exact", length=200.0, width=20.0, tilt=35.0, name="flume262k_exact"),
        # the polydisperse hopper, funnel and flume: every boundary routine, the largest plain run
        _case("step", 524288, 20, layout="funnel", spread=0.2, name="funnel524k_fast"),
        # an ensemble of uneven flumes with their own materials and slopes, 64 steps a call
        _case("step", 64, 64, layout="ensemble", flumes=64, name="ensemble64_fast"),
        # filling the hopper: a pile on the closed door, odd count
        _case("step", 20011, 50, layout="fill", mode="exact", name="fill20k_exact"),
        # a driver that keeps the particles on the host: one step a call
        _case("host", 100003, 1, length=200.0, width=20.0, tilt=35.0, name="host100k_fast"),
        # the reference's loop, one entry point per routine
        _case("routines", 8192, 4, mode="exact", name="routines8k"),
        # gradients of the deposit centroid with respect to materials and the initial state
        _case("adjoint", 32768, 100, mode="exact", friction="dev", length=80.0, tilt=35.0, name="adjoint32k"),
    ]


def draw(rng):
    """A case of the same ranges: counts spread over their logarithm, odd ones among them."""
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def geometry(n):
        if n <= 16384:
            return {"length": 40.0, "width": 4.0}
        return {"length": 80.0, "width": 4.0} if n <= 65536 else {"length": 200.0, "width": 20.0}

    kind = rng.choice(["step"] * 6 + ["funnel", "fill", "ensemble", "host", "routines", "adjoint"])
    mode, friction = rng.choice(["fast", "exact"]), rng.choice(["hst", "dev"])
    tilt = round(rng.uniform(25.0, 40.0), 3)
    if kind == "step":
        n = logint(256, 262144)
        k = max(8, min(logint(16, 400), 5_000_000 // n))
        return _case("step", n, k, mode=mode, friction=friction, tilt=tilt, **geometry(n))
    if kind == "funnel":
        n = logint(4096, 262144)
        return _case("step", n, max(8, min(logint(10, 60), 4_000_000 // n)), layout="funnel", mode=mode,
                     friction=friction, spread=round(rng.uniform(0.05, 0.2), 3))
    if kind == "fill":
        n = logint(1024, 65536)
        return _case("step", n, logint(10, 60), layout="fill", mode=mode, friction=friction, tilt=tilt)
    if kind == "ensemble":
        f = logint(4, 64)
        return _case("step", f, logint(8, 64), layout="ensemble", flumes=f, mode=mode, friction=friction)
    if kind == "host":
        n = logint(2048, 262144)
        return _case("host", n, 1, mode=mode, friction=friction, tilt=tilt, **geometry(n))
    if kind == "routines":
        return _case("routines", logint(512, 32768), rng.randint(1, 5), mode="exact", friction=friction, tilt=tilt)
    # counts of the adjoint are multiples of 8, which puts the records of its tape on 64-byte boundaries
    return _case("adjoint", 8 * logint(128, 4096), logint(20, 100), mode="exact", friction=friction, tilt=tilt,
                 length=80.0)


# ------------------------------------------------------------------ inputs

def _inputs(case, seed):
    """(system_par, Funnel, particles, phase, ntags) of a case: arrays over flumes for an ensemble.
    The clumps rest on each other with loaded contacts (pressed 2e-5 cm into their supports)."""
    rng = np.random.default_rng(seed)
    geo = {"seed": 20240613 + 7919 * (seed % 100003), "tilt_deg": case["tilt"], "overlap": 2.0e-5}
    phase, ntags = PHASE_AVALANCHE, 9
    if case["layout"] == "ensemble":
        cfgs = ensemble_configs(case["flumes"], layout="bed", overlap=2.0e-5)
        sys, fun, pp = ensemble_state([dataclasses.replace(c, seed=c.seed + 613 * (seed % 100003)) for c in cfgs])
        cost, sint = (np.repeat(sys[k], sys["npart"]) for k in ("cost", "sint"))
    else:
        if case["layout"] == "funnel":
            cfg = funnel_524k(**{**geo, "n": case["n"], "size_spread": case["spread"]})
            ntags = cfg.ntags
        else:
            cfg = flume_2k(n=case["n"], width=case["width"], Lflume=case["length"],
                           layout="pile" if case["layout"] == "fill" else "bed", **geo)
        sys, fun, pp = flume_state(cfg)
        cost, sint = float(sys["cost"]), float(sys["sint"])
    n = len(pp)
    if case["layout"] == "fill":
        # the pile on the closed door a second before it opens, still settling
        phase = PHASE_FILL
        sys["time"] = -1.0
        sys["side"][0] = 15.0
        pp["vv"][:, 2] = -15.0
    else:
        z = pp["rrot"][:, 2]
        u = 110.0 * (0.5 + 0.5 * z / max(1e-9, float(z.max())))
        pp["vv"][:, 0] = u * cost
        pp["vv"][:, 2] = -u * sint
        if case["layout"] == "funnel":   # the hopper's half falls through the open door
            pp["vv"][:n // 2] = (0.0, 0.0, -25.0)
    pp["vv"] += 4.0 * rng.standard_normal((n, 3))
    pp["ww"] = 30.0 * rng.standard_normal((n, 3))
    return sys, fun, pp, phase, ntags


def _pinned(n):
    """Page-locked host arrays as a program that copies every so often keeps them: particles, a, alpha."""
    t = [torch.empty(max(1, n) * PARTICLE.itemsize, dtype=torch.uint8, pin_memory=True)]
    t += [torch.empty(max(1, 3 * n), dtype=torch.float64, pin_memory=True) for _ in range(2)]
    return t, [t[0].numpy().view(PARTICLE)[:n]] + [x.numpy()[:3 * n].reshape(n, 3) for x in t[1:]]


def _ptr(a):
    return a.ctypes.data_as(C.c_void_p)


def _check(status, what):
    if status != 0:
        raise RuntimeError("%s failed: %d" % (what, status))


class _State:
    """A context with the particles of a case in host memory, where the call starts from."""

    def __init__(self, case, seed):
        sys, fun, pp, phase, ntags = _inputs(case, seed)
        self.call, self.steps, self.n = case["call"], case["steps"], len(pp)
        self.eng = Engine(sys, fun, ntags=ntags, phase=phase,
                          friction=FRICTION_DEV if case["friction"] == "dev" else FRICTION_HST,
                          fp_mode=FP_FAST if case["mode"] == "fast" else FP_EXACT)
        self.keep_in, self.src = _pinned(self.n)
        self.keep_out, self.out = _pinned(self.n)
        self.src[0][:] = pp
        if self.call == "adjoint":
            return
        # the accelerations a run starts from (the program's start-up force pass)
        self.eng.import_particles(pp)
        self.eng.forces()
        self.eng.swap_accel()
        self.src[0][:], self.src[1][:], self.src[2][:] = self.eng.export_particles()
        self.handle = C.c_void_p(self.eng._h.value)


def prepare(case, seed):
    return _State(case, seed)


# ------------------------------------------------------------------ the calls

def run(s):
    if s.call == "adjoint":
        s.eng.import_particles(s.src[0])
        return s.eng.adjoint(s.steps, 500)
    L, src, out = lib(), s.src, s.out
    if s.call == "host":
        s.eng.step_host(src[0], src[1], src[2], out[0], out[1], out[2])
    else:
        _check(L.af3d_import_particles(s.handle, _ptr(src[0]), _ptr(src[1]), _ptr(src[2])), "import")
        if s.call == "step":
            _check(L.af3d_step(s.handle, s.steps), "step")
        else:
            e = s.eng
            for _ in range(s.steps):
                e.init_verlet()
                e.advance_time()
                e.rotate_vectors()
                e.clear_forces()
                e.cell_build()
                for nw in range(3):
                    e.force_hop(nw)
                e.force_funnel()
                e.force_fcorners()
                e.force_walls()
                e.force_part(0)
                e.force_flume()
                e.get_accel()
                e.finish_verlet()
                e.swap_accel()
        _check(L.af3d_export_particles(s.handle, _ptr(out[0]), _ptr(out[1]), _ptr(out[2])), "export")
    return {**{f: out[0][f] for f in FIELDS}, "a": out[1], "alpha": out[2]}


def work(case):
    """Per step a clump's state is read and written once (192 + 32 read, 192 written, 32 of cell
    list) and its FP64 arithmetic done (the predictor, one sphere contact, the accelerations);
    the host arrays cross once each way.  The adjoint writes and reads its tape (540 B) as well
    and does about three times the arithmetic."""
    n = case["n"]
    if case["layout"] == "ensemble":
        n = sum(c.n for c in ensemble_configs(case["flumes"]))
    ns = float(n) * case["steps"]
    io = 2.0 * (PARTICLE.itemsize + 48) * n
    if case["call"] == "adjoint":
        return {"bytes": ns * (2 * 448 + 2 * 540) + 2 * io, "flops": 3 * 441 * ns}
    return {"bytes": ns * 448 + io, "flops": 441 * ns}


# ------------------------------------------------------------------ the same in plain 64-bit torch

GYR, SPH_FACT, ROOT2, DRAG, GRAV = 4.4494897427831781, 4.188790204786391, 1.414213562373095, 1.895e-3, 981.0
HOP_H, HOP_W, YL, YR, YFUN, LFUN = 25.0, 15.0, 7.5, 22.5, 30.0, 70.0
CORNERS = ((1, 1, 1), (1, -1, -1), (-1, -1, 1), (-1, 1, -1))


def _dot(a, b):
    p = a * b
    return p[..., 0] + p[..., 1] + p[..., 2]


def _v(x, y, z):
    return torch.stack(torch.broadcast_tensors(x, y, z), -1)


class _Model:
    """Clumps of all flumes in one set of arrays; P holds each clump's own parameters."""

    def __init__(self, case, seed):
        sys, fun, pp, phase, _ = _inputs(case, seed)
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)
        sys_a, fun_a = np.atleast_1d(sys), np.atleast_1d(fun)
        self.fl = torch.tensor(np.repeat(np.arange(len(sys_a)), sys_a["npart"]), device=dev)
        self.par = {k: t(sys_a[k]) for k in ADJ_PARAMS}
        own = {k: t(sys_a[k]) for k in ("sint", "cost", "dy2", "fr_fact_pp", "fr_fact_pw")}
        own["side_y"] = t(sys_a["side"][:, 1])
        own.update({k: t(fun_a[k]) for k in ("sinfi", "cosfi", "tanfi")})
        self.P = {k: x[self.fl] for k, x in own.items()}
        self.dt, self.hdt = float(sys_a["dt"][0]), float(sys_a["hdt"][0])
        self.time = float(sys_a["time"][0])
        self.fill, self.dev_law = phase == PHASE_FILL, case["friction"] == "dev"
        self.rad, self.mass, self.I = t(pp["radius"]), t(pp["mass"]), t(pp["moment_of_inertia"][:, 0])
        self.msph = SPH_FACT * t(pp["density"]) * self.rad ** 3
        self.r, self.v, self.w = t(pp["rr"]), t(pp["vv"]), t(pp["ww"])
        self.R = torch.stack([t(pp[f]) for f in ("Rmatx", "Rmaty", "Rmatz")], 1)
        self.s = t(pp["rr_s"])
        self.corners = torch.tensor(CORNERS, dtype=torch.float64, device=dev)
        self.a, self.al = torch.zeros_like(self.r), torch.zeros_like(self.r)
        self.pairs = self.candidates(skin=0.03)

    def centres(self):
        return self.r[:, None] + (self.rad / ROOT2)[:, None, None] * torch.einsum("nij,kj->nki", self.R, self.corners)

    def candidates(self, skin):
        """Ordered sphere pairs of different clumps that may touch while no two approach by `skin`."""
        r, fl, n = self.r, self.fl, len(self.r)
        reach = GYR * float(self.rad.max()) + skin
        c = torch.floor((r - r.min(0).values) / reach).long() + 1
        dim = c.max(0).values + 2
        key = ((fl * dim[2] + c[:, 2]) * dim[1] + c[:, 1]) * dim[0] + c[:, 0]
        skey, order = key.sort()
        found = []
        for dz in (-1, 0, 1):
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    nk = key + (dz * dim[1] + dy) * dim[0] + dx
                    lo, hi = torch.searchsorted(skey, nk), torch.searchsorted(skey, nk, right=True)
                    for q in range(int((hi - lo).max())):
                        i = torch.nonzero(lo + q < hi).squeeze(1)
                        j = order[lo[i] + q]
                        lim = 0.5 * GYR * (self.rad[i] + self.rad[j]) + skin
                        keep = (i != j) & ((r[i] - r[j]).square().sum(1) < lim * lim)
                        found.append(torch.stack([i[keep], j[keep]]))
        i, j = torch.cat(found, 1)
        out = []
        for k in range(4):
            for m in range(4):
                lim = self.rad[i] + self.rad[j] + skin
                near = (self.s[j, m] - self.s[i, k]).square().sum(1) < lim * lim
                ii = i[near]
                out.append(torch.stack([ii, j[near], torch.full_like(ii, k), torch.full_like(ii, m)]))
        return torch.cat(out, 1)

    def law(self, i, dv, n, comp, km, gm, mass, mu, cns, arm, xi0, gate):
        """Adds the contacts' forces and torques to the sums of their owners i."""
        vn = _dot(dv, n)
        vt = dv - vn[:, None] * n
        normal = km * comp - gm * vn
        on = torch.nonzero(~(normal <= 0) if gate else normal > 0).squeeze(1)
        i, dv, n, normal, vt, mass, mu, cns, arm = (x[on] for x in (i, dv, n, normal, vt, mass, mu, cns, arm))
        slide = _dot(vt, vt) > 0
        vtm = torch.where(slide, _dot(vt, vt), torch.ones_like(normal)).sqrt()
        xi = self.dt * _dot(dv, vt / vtm[:, None])
        xi = torch.where(cns * normal < xi.abs(), torch.zeros_like(xi), xi)
        fs = 1.0e12 * mass * xi + 2.0e6 * mass * (xi / self.dt)
        coul = (fs.abs() > mu * normal) | (xi == 0 if xi0 else torch.zeros_like(slide))
        af = 0.8 * mu * normal / vtm
        af = af / (1.0 + (self.dt * af / mass) ** 2)
        g = torch.where(slide, torch.where(coul, af, fs / vtm), torch.zeros_like(af))
        f = g[:, None] * vt - normal[:, None] * n
        self.F = self.F.index_add(0, i, f)
        self.T = self.T.index_add(0, i, torch.linalg.cross(arm, f))

    def par_of(self, name, i):
        return self.par[name][self.fl[i]]

    def wall(self, hit, k, point, normal, comp, gate=False):
        """Wall contacts of sphere k of the clumps where `hit`."""
        i = torch.nonzero(hit).squeeze(1)
        arm = point[i] - self.r[i]
        m = self.msph[i]
        self.law(i, -(self.v[i] + torch.linalg.cross(self.w[i], arm)), normal[i], comp[i],
                 0.5 * self.par_of("kappa_pw", i) * m, 0.5 * self.par_of("gamma_pw", i) * m, m,
                 self.par_of("mu_pw", i), self.P["fr_fact_pw"][i], arm, True, gate)

    def either(self, k, first, second):
        """Two facing walls, of which the second wins: each is (hit, contact point, normal, compression)."""
        (h1, p1, n1, c1), (h2, p2, n2, c2) = first, second
        pick = h2[:, None]
        self.wall(h1 | h2, k, torch.where(pick, p2, p1), torch.where(pick, n2, n1), torch.where(h2, c2, c1))

    def hopper(self):
        one, nil = torch.ones_like(self.rad), torch.zeros_like(self.rad)
        for k in range(4):
            x, y, z = self.s[:, k].unbind(1)
            inside = ~((z < HOP_H) | (x > HOP_W))
            hit = lambda d: inside & (d <= self.rad)
            self.either(k, (hit(x), _v(nil, y, z), _v(-one, nil, nil), self.rad - x),
                        (hit(HOP_W - x), _v(HOP_W * one, y, z), _v(one, nil, nil), self.rad - (HOP_W - x)))
            self.either(k, (hit(y - YL), _v(x, YL * one, z), _v(nil, -one, nil), self.rad - (y - YL)),
                        (hit(YR - y), _v(x, YR * one, z), _v(nil, one, nil), self.rad - (YR - y)))
            if self.time < 0:
                self.wall(hit(z - HOP_H), k, _v(x, y, HOP_H * one), _v(nil, nil, -one), self.rad - (z - HOP_H))

    def slope(self, p):
        c, s = self.P["cost"], self.P["sint"]
        return p[:, 0] * c - p[:, 2] * s, p[:, 1], p[:, 0] * s + p[:, 2] * c

    def lab(self, x, y, z):
        c, s = self.P["cost"], self.P["sint"]
        return _v(x * c + z * s, y, z * c - x * s)

    def chute(self):
        """Funnel walls, funnel corners and the flume's side walls."""
        P, rad, nil = self.P, self.rad, torch.zeros_like(self.rad)
        one = torch.ones_like(rad)
        si, co, ta = P["sinfi"], P["cosfi"], P["tanfi"]
        for k in range(4):
            x, y, z = self.slope(self.s[:, k])
            up = ~(x > LFUN - rad * si)
            d1, d2 = (y - x * ta).abs() * co, (YFUN - y - x * ta).abs() * co
            self.either(k, (up & (d1 <= rad), self.lab(x + d1 * si, y - d1 * co, z), self.lab(si, -co, nil), rad - d1),
                        (up & (d2 <= rad), self.lab(x + d2 * si, y + d2 * co, z), self.lab(si, co, nil), rad - d2))
        for k in range(4):
            x, y, z = self.slope(self.s[:, k])
            lo, hi = P["dy2"], P["side_y"] + P["dy2"]
            dx = LFUN - x
            dy = torch.where(y <= P["dy2"] + P["side_y"] / 2, lo, hi) - y
            d2 = dx * dx + dy * dy
            hit = ~((x < LFUN - rad * si) | (x > LFUN + rad) | (y > hi) | (y < lo) | (d2 > rad * rad))
            d = torch.where(hit, d2, one).sqrt()
            nx, ny = dx / d, dy / d
            self.wall(hit, k, self.lab(x + rad * nx, y + rad * ny, z), self.lab(nx, ny, nil), rad - d, gate=True)
        for k in range(4):
            q = self.s[:, k]
            x, y, z = q.unbind(1)
            down = self.slope(q)[0] > LFUN
            lo, hi = P["dy2"], P["side_y"] + P["dy2"]
            self.either(k, (down & (y - lo <= rad), _v(x, lo, z), _v(nil, -one, nil), rad - (y - lo)),
                        (down & (hi - y <= rad), _v(x, hi, z), _v(nil, one, nil), rad - (hi - y)))

    def bed(self):
        c, s = self.P["cost"], self.P["sint"]
        for k in range(4):
            x, y, z = self.s[:, k].unbind(1)
            d = (c * (-(s / c) * x - z)).abs()
            self.wall(d <= self.rad, k, _v(x - d * s, y, z - d * c), _v(-s, torch.zeros_like(s), -c), self.rad - d)

    def particles(self):
        i, j, k, m = self.pairs
        d = self.s[j, m] - self.s[i, k]
        sep = self.rad[i] + self.rad[j]
        hit = _dot(d, d).detach() < sep * sep
        i, j, k, d, sep = i[hit], j[hit], k[hit], d[hit], sep[hit]
        dist = _dot(d, d).sqrt()
        n = d / dist[:, None]
        at = self.s[i, k] + self.rad[i][:, None] * n
        arm = at - self.r[i]
        dv = (self.v[j] + torch.linalg.cross(self.w[j], at - self.r[j])) - (
            self.v[i] + torch.linalg.cross(self.w[i], arm))
        meff = 0.5 * (self.msph[j] + self.msph[i])
        self.law(i, dv, n, sep - dist, 0.5 * self.par_of("kappa_pp", i) * meff,
                 0.5 * self.par_of("gamma_pp", i) * meff, self.msph[i], self.par_of("mu_pp", i),
                 self.P["fr_fact_pp"][i], arm, self.dev_law, False)

    def forces(self):
        self.F, self.T = torch.zeros_like(self.r), torch.zeros_like(self.r)
        if self.fill:
            self.particles()
            self.hopper()
        else:
            self.hopper()
            self.chute()
            self.particles()
            self.bed()
        speed = _dot(self.v, self.v).sqrt()
        drag = DRAG * self.rad * self.rad / self.mass * speed
        down = torch.tensor([0.0, 0.0, GRAV], dtype=torch.float64, device=self.r.device)
        a = self.F / self.mass[:, None] - drag[:, None] * self.v - down
        body = torch.einsum("nij,ni->nj", self.R, self.T) / self.I[:, None]
        return a, torch.einsum("nij,nj->ni", self.R, body)

    def step(self):
        dt, hdt = self.dt, self.hdt
        self.r = self.r + dt * (self.v + hdt * self.a)
        turn = dt * (self.w + hdt * self.al)
        self.v, self.w = self.v + dt * self.a, self.w + dt * self.al
        ang = _dot(turn, turn).sqrt()
        u = turn / ang[:, None]
        sn, omc = torch.sin(ang)[:, None, None], 2.0 * (torch.sin(0.5 * ang) ** 2)[:, None, None]
        nil = torch.zeros_like(ang)
        x, y, z = u.unbind(1)
        K = torch.stack([nil, -z, y, z, nil, -x, -y, x, nil], 1).view(-1, 3, 3)
        R = self.R + sn * (K @ self.R) + omc * (K @ (K @ self.R))
        self.R = R / R.square().sum(1, keepdim=True).sqrt()
        self.s = self.centres()
        self.time = self.time + dt
        a, al = self.forces()
        self.v, self.w = self.v + hdt * (a - self.a), self.w + hdt * (al - self.al)
        self.a, self.al = a, al


def exact(case, seed):
    m = _Model(case, seed)
    if case["call"] == "adjoint":
        leaves = [m.r, m.v, m.w, m.R] + [m.par[k] for k in ADJ_PARAMS]
        for x in leaves:
            x.requires_grad_(True)
        m.s = m.centres()
        m.a, m.al = m.forces()
        for _ in range(case["steps"]):
            m.step()
        J = (m.mass * m.slope(m.r)[0]).sum() / m.mass.sum()
        g = [x.detach().cpu().numpy() for x in torch.autograd.grad(J, leaves)]
        return {"J": float(J.detach()), "r0": g[0], "v0": g[1], "w0": g[2], "R0": g[3],
                "params": {k: float(x[0]) for k, x in zip(ADJ_PARAMS, g[4:])}}
    with torch.no_grad():
        m.a, m.al = m.forces()
        for _ in range(case["steps"]):
            m.step()
    out = dict(zip(FIELDS, (m.r, m.v, m.w, m.R[:, 0], m.R[:, 1], m.R[:, 2], m.s)), a=m.a, alpha=m.al)
    return {k: x.cpu().numpy() for k, x in out.items()}
