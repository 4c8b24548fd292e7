"""The work that a user of this library has it do, as cases of a measurement:
listed() and draw() name them, prepare() makes what a program holds before
the call, run() is one pass through the public entry points, work() the bytes
and operations a pass cannot do without, exact() the outputs in plain 64-bit
torch arithmetic.

Kinds of case:

    bodies   the states of all 27 bodies at n times (batch.bodies_device)
    forces   the accelerations of n particles, each at its own time, with or
             without six variational particles each (batch.forces_device)
    shared   the accelerations of n particles at one time
             (batch.forces_shared_time_device)
    dropin   one REBOUND simulation with ASSIST attached, integrated forward:
             host particles in, host particles out (Simulation.integrate)
    batch    n independent particles with their own spans
             (batch.integrate_batch_device), with or without variational
             particles, with or without dense output
"""
import atexit
import ctypes
import math
import shutil
import struct
import tempfile

import numpy as np
import torch

from assist_gb300 import Ephem, Extras, Simulation, batch, synth

T0 = 8000.0                          # start of every integration (days from JD 2451545.0)
T_BEG, T_END = 7900.0, 9200.0        # the ephemeris's span
N_BODY = 27                          # Sun, planets, Moon, Pluto, 16 asteroids

# Algorithmic operations, counted once per add, multiply, divide and square
# root: the body states and the particle-independent parts of the force terms
# at one time, a particle's force terms, the six variational accelerations,
# IAS15's own work per evaluation and per step, and per-component numbers of
# evaluations per day for a shared or own adaptive step (measured means of
# the populations below).
OPS_TABLE, OPS_FORCE, OPS_VAR, OPS_IAS_EVAL, OPS_IAS_STEP = 3521, 907, 1500, 150, 294
OPS_BODIES = 4200
EVALS_PER_DAY = {"mba": 1.4, "neo": 3.0, "mix": 1.9}


def listed():
    return [
        # where the planets are at an epoch: one lookup
        {"name": "bodies-1", "kind": "bodies", "n": 1},
        # an ephemeris table for many observation times
        {"name": "bodies-30011", "kind": "bodies", "n": 30011},
        # the force model called from a user's own integrator on a few objects
        {"name": "forces-33", "kind": "forces", "n": 33, "var": False, "nongrav": 0.0},
        # the force model over a catalogue, a tenth of it with A1, A2
        {"name": "forces-100003", "kind": "forces", "n": 100003, "var": False, "nongrav": 0.1},
        # the same with partial derivatives, for orbit fits
        {"name": "forces-var-20011", "kind": "forces", "n": 20011, "var": True, "nongrav": 0.1},
        # a catalogue's accelerations at one epoch
        {"name": "shared-20011", "kind": "shared", "n": 20011, "nongrav": 0.1},
        # the reference's own use: a few objects in one simulation
        {"name": "dropin-3", "kind": "dropin", "pop": "mba", "n": 3, "days": 120.0, "var": 0},
        # a thousand main-belt objects in one simulation for a year
        {"name": "dropin-1024", "kind": "dropin", "pop": "mba", "n": 1024, "days": 365.25, "var": 0},
        # near-Earth objects with their state transition matrices
        {"name": "dropin-neo-var-70", "kind": "dropin", "pop": "neo", "n": 70, "days": 60.0, "var": 6},
        # observers' ephemerides of a few hundred objects every ten days,
        # planets from an SPK kernel
        {"name": "batch-dense-200", "kind": "batch", "pop": "mix", "n": 200, "days": 200.0, "spread": 1.0,
         "var": False, "nongrav": 0.1, "every": 10.0, "planets": "spk"},
        # a survey's catalogue over a year
        {"name": "batch-65536", "kind": "batch", "pop": "mix", "n": 65536, "days": 365.25, "spread": 1.0,
         "var": False, "nongrav": 0.1, "every": 0.0, "planets": "440"},
        # orbit fits over arcs of a month to two years
        {"name": "batch-var-2053", "kind": "batch", "pop": "mix", "n": 2053, "days": 730.0, "spread": 24.0,
         "var": True, "nongrav": 0.1, "every": 0.0, "planets": "440"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["bodies", "forces", "forces", "shared", "dropin", "dropin", "batch", "batch", "batch"])
    if kind == "bodies":
        return {"kind": kind, "n": _log_int(rng, 1, 30011)}
    if kind == "forces":
        var = rng.random() < 0.4
        return {"kind": kind, "n": _log_int(rng, 1, 20011 if var else 100003), "var": var,
                "nongrav": rng.choice([0.0, 0.1, 1.0])}
    if kind == "shared":
        return {"kind": kind, "n": _log_int(rng, 1, 20011), "nongrav": rng.choice([0.0, 0.1])}
    if kind == "dropin":
        var = rng.choice([0, 0, 6])
        return {"kind": kind, "pop": rng.choice(["mba", "neo"]), "n": _log_int(rng, 1, 150 if var else 1500),
                "days": round(math.exp(rng.uniform(math.log(20.0), math.log(200.0))), 3), "var": var}
    var = rng.random() < 0.3
    dense = not var and rng.random() < 0.4
    return {"kind": kind, "pop": rng.choice(["mba", "mix", "mix"]), "n": _log_int(rng, 3, 2053 if var else 30000),
            "days": 10.0 * rng.randint(3, 36), "spread": 1.0 if dense else rng.choice([1.0, 12.0]), "var": var,
            "nongrav": rng.choice([0.0, 0.1]), "every": 10.0 if dense else 0.0, "planets": rng.choice(["440", "440", "spk"])}


# ------------------------------------------------------------------ inputs

class _World:
    """The ephemeris files and handles every case shares, made on first use."""
    _one = None

    def __init__(self):
        self.dir = tempfile.mkdtemp(prefix="assist_gb300_cases_")
        atexit.register(shutil.rmtree, self.dir, True)
        self.planets, self.asteroids, self.system = synth.write_ephemeris(self.dir, t_beg=T_BEG, t_end=T_END)
        self.spk = synth.write_planets_spk(self.dir, self.system, 1, T_BEG, T_END)
        self._ephem = {}
        self._plain = None

    @classmethod
    def get(cls):
        if cls._one is None:
            cls._one = cls()
        return cls._one

    def ephem(self, planets="440"):
        if planets not in self._ephem:
            self._ephem[planets] = Ephem(self.planets if planets == "440" else self.spk, self.asteroids)
        return self._ephem[planets]

    def plain(self):
        if self._plain is None:
            self._plain = _PlainEphem(self.planets, self.asteroids)
        return self._plain


def _clear_of_planets(system, state, days, limit=0.02):
    """Which particles keep `limit` AU away from the Earth, Mars and (twice
    that) Jupiter over `days` on their two-body orbits: the others' end states
    hang on the last bit of every operation, and no two correct programs give
    the same ones."""
    dev, f8 = "cuda", torch.float64
    sp, sv = system.sun(np.array(T0))
    r = torch.tensor(state[:, :3] - sp, dtype=f8, device=dev)
    v = torch.tensor(state[:, 3:] - sv, dtype=f8, device=dev)
    mu = synth.GMS
    rn = r.norm(dim=1)
    rv = (r * v).sum(1)
    a = 1.0 / (2.0 / rn - (v * v).sum(1) / mu)
    ev = ((v * v).sum(1, keepdim=True) - mu / rn[:, None]) * r / mu - rv[:, None] * v / mu
    e = ev.norm(dim=1)
    h = torch.linalg.cross(r, v)
    p = ev / e[:, None]
    q = torch.linalg.cross(h, p) / h.norm(dim=1, keepdim=True)
    ea = torch.atan2(rv / torch.sqrt(mu * a), 1.0 - rn / a)
    m0 = ea - e * torch.sin(ea)
    n = torch.sqrt(mu / a ** 3)
    b = a * torch.sqrt(1.0 - e * e)
    ok = torch.ones(len(state), dtype=torch.bool, device=dev)
    ts = np.linspace(T0, T0 + days, max(2, int(days / 0.5)) + 1)
    sun = system.sun(ts)[0]
    bodies = [(torch.tensor(system.body(i, ts)[0] - sun, dtype=f8, device=dev), d)
              for i, d in ((3, limit), (5, limit), (6, 2.0 * limit))]
    step = max(1, 4_000_000 // max(1, len(state)))
    for k in range(0, len(ts), step):
        dt = torch.tensor(ts[k:k + step] - T0, dtype=f8, device=dev)[:, None]
        m = torch.remainder(m0 + n * dt, 2.0 * math.pi)
        x = m + e * torch.sin(m)
        for _ in range(6):
            x = x - (x - e * torch.sin(x) - m) / (1.0 - e * torch.cos(x))
        pos = (a * (torch.cos(x) - e))[..., None] * p + (b * torch.sin(x))[..., None] * q
        for w, d in bodies:
            ok &= ((pos - w[k:k + step, None, :]).norm(dim=2) > d).all(0)
    return ok.cpu().numpy()


def _population(kind, n, seed, days, nongrav):
    """n particles of the population that keep clear of the planets."""
    system = _World.get().system
    want = n + max(8, n // 4)
    pop = synth.population(system, kind, want, seed=seed, t0=T0, length=days, nongrav_frac=nongrav)
    keep = np.nonzero(_clear_of_planets(system, pop.state, days))[0][:n]
    if len(keep) < n:
        raise RuntimeError("population: %d of %d particles are clear of the planets" % (len(keep), n))
    return pop.state[keep], pop.params[keep]


def _spans(case, seed):
    """Lengths of a batch case: equal, or log-uniform down to days / spread."""
    days, spread = case["days"], case["spread"]
    if spread == 1.0:
        return np.full(case["n"], days)
    u = np.random.default_rng(seed + 77).uniform(0.0, 1.0, case["n"])
    return days * np.exp(-u * math.log(spread))


def _inputs(case, seed):
    """The case's inputs as numpy arrays: all that prepare() and exact() start from."""
    kind, n = case["kind"], case["n"]
    rng = np.random.default_rng(seed + 13)
    if kind == "bodies":
        return {"t": rng.uniform(T_BEG + 1.0, T_END - 1.0, n)}
    if kind in ("forces", "shared"):
        pop = synth.population(_World.get().system, "mix", n, seed=seed, t0=T0, length=1.0,
                               nongrav_frac=case["nongrav"])
        t = T0 + rng.uniform(-40.0, 40.0, n if kind == "forces" else 1)
        got = {"t": t, "state": pop.state, "params": pop.params if case["nongrav"] else None}
        if case.get("var"):
            got["var"] = np.eye(6) + 1e-3 * rng.standard_normal((n, 6, 6))
        return got
    if kind == "dropin":
        state, _ = _population(case["pop"], n, seed, case["days"], 0.0)
        return {"state": state}
    state, params = _population(case["pop"], n, seed, case["days"], case["nongrav"])
    got = {"state": state, "params": params if case["nongrav"] else None, "span": _spans(case, seed)}
    if case["every"]:
        got["out"] = T0 + case["every"] * np.arange(1, int(round(case["days"] / case["every"])) + 1)
    return got


def _gpu(a):
    return None if a is None else torch.tensor(a, dtype=torch.float64, device="cuda")


def prepare(case, seed):
    x = _inputs(case, seed)
    kind, n = case["kind"], case["n"]
    s = {"kind": kind, "ephem": _World.get().ephem(case.get("planets", "440"))}
    if kind == "bodies":
        s["t"] = _gpu(x["t"])
    elif kind == "forces":
        s.update(t=_gpu(x["t"]), state=_gpu(x["state"]), params=_gpu(x["params"]), var=_gpu(x.get("var")))
    elif kind == "shared":
        s.update(t=float(x["t"][0]), state=_gpu(x["state"]), params=_gpu(x["params"]))
    elif kind == "dropin":
        sim = Simulation.create()
        s.update(sim=sim, extras=Extras(sim, s["ephem"]), end=T0 + case["days"])
        for p in x["state"]:
            sim.add(*p)
        for i in range(n if case["var"] else 0):
            for k, name in enumerate(("x", "y", "z", "vx", "vy", "vz")):
                setattr(sim.particle(sim.add_variation(i)), name, 1.0)
        s["start"] = np.array(_particles(sim))
        s["dt"] = sim.dt
    else:
        s.update(t0=torch.full((n,), T0, dtype=torch.float64, device="cuda"), t_end=_gpu(T0 + x["span"]),
                 state=_gpu(x["state"]), params=_gpu(x["params"]))
        if case["var"]:
            s["var"] = torch.eye(6, dtype=torch.float64, device="cuda").repeat(n, 1, 1)
        if case["every"]:
            k = len(x["out"])
            s["out_start"] = torch.arange(0, n * k + 1, k, dtype=torch.int32, device="cuda")
            s["out_t"] = _gpu(np.tile(x["out"], n))
    return s


def _particles(sim):
    """The simulation's particle array (REBOUND's struct reb_particle, sixteen
    8-byte words each, position and velocity first) without a copy."""
    p = ctypes.cast(sim._particles, ctypes.POINTER(ctypes.c_double))
    return np.ctypeslib.as_array(p, (sim.N, 16))[:, :6]


def run(s):
    kind = s["kind"]
    if kind == "bodies":
        return batch.bodies_device(s["ephem"], s["t"])
    if kind == "forces":
        acc, var_acc = batch.forces_device(s["ephem"], s["t"], s["state"], params=s["params"], var_state=s["var"])
        return {"acc": acc, "var_acc": var_acc} if var_acc is not None else {"acc": acc}
    if kind == "shared":
        return batch.forces_shared_time_device(s["ephem"], s["t"], s["state"], params=s["params"])
    if kind == "dropin":
        # the same start again: positions, time and first step
        sim = s["sim"]
        p = _particles(sim)
        p[:] = s["start"]
        sim.t, sim.dt = T0, s["dt"]
        if sim.integrate(s["end"]) != 0:
            raise RuntimeError("integration failed: status %d" % sim.status)
        return p.copy()
    state, status = s["state"].clone(), torch.empty(len(s["state"]), dtype=torch.int32, device="cuda")
    out = {"state": state, "status": status}
    if "out_t" in s:
        out["dense"] = torch.empty((len(s["out_t"]), 6), dtype=torch.float64, device="cuda")
        batch.integrate_batch_dense_device(s["ephem"], s["t0"], s["t_end"], state, s["out_start"], s["out_t"],
                                           out["dense"], params=s["params"], status=status)
    else:
        if "var" in s:
            out["var"] = s["var"].clone()
        batch.integrate_batch_device(s["ephem"], s["t0"], s["t_end"], state, params=s["params"],
                                     var_state=out.get("var"), status=status)
    return out


def work(case):
    kind, n = case["kind"], case["n"]
    if kind == "bodies":
        return {"bytes": 8.0 * n * (1 + 10 * N_BODY), "flops": float(OPS_BODIES) * n}
    if kind == "forces":
        var = 6 if case["var"] else 0
        return {"bytes": 8.0 * n * (1 + 6 + 3 + 9 * var + (3 if case["nongrav"] else 0)),
                "flops": float(n) * (OPS_TABLE + OPS_FORCE + (OPS_VAR if var else 0))}
    if kind == "shared":
        return {"bytes": 8.0 * n * (9 + (3 if case["nongrav"] else 0)), "flops": float(n) * OPS_FORCE + OPS_TABLE}
    pop = case["pop"]
    evals = EVALS_PER_DAY[pop] * case["days"]
    if kind == "batch" and case["spread"] > 1.0:
        evals *= (1.0 - 1.0 / case["spread"]) / math.log(case["spread"])     # mean of the log-uniform lengths
    each = OPS_FORCE + OPS_IAS_EVAL + OPS_IAS_STEP / 20.0
    if case["var"]:
        each += OPS_VAR + 6 * OPS_IAS_EVAL
    steps = evals / 20.0
    tables = 8.0 * steps * (1.0 if kind == "dropin" else n / 32.0)
    outs = int(round(case["days"] / case["every"])) if case.get("every") else 0
    return {"bytes": 8.0 * n * (12 + 7 * outs + (72 if case["var"] else 0)),
            "flops": float(n) * evals * each + tables * OPS_TABLE}


# ------------------------------------------------------------------ plain 64-bit arithmetic

class _PlainEphem:
    """The ephemeris files read and evaluated with torch in 64 bits."""
    COLUMNS = 11                      # Mercury .. Pluto, Moon, Sun

    def __init__(self, planets, asteroids):
        raw = open(planets, "rb").read()
        self.beg, _, self.inc, n_con = struct.unpack_from("<dddi", raw, 0xA5C)
        self.au, self.emrat = struct.unpack_from("<dd", raw, 0xA5C + 28)
        cols = [struct.unpack_from("<iii", raw, 0xA5C + 44 + 12 * c) for c in range(self.COLUMNS)]
        words = 2 + max(o - 3 + 3 * c * i for o, c, i in cols)
        words = max(words, 2 + sum(c * i * m for c, i, m in synth.LAYOUT))
        names = [raw[0xFC + 6 * k:0xFC + 6 * k + 6].decode().strip() for k in range(min(n_con, 400))]
        vals = np.frombuffer(raw, "<f8", n_con, 8 * words)
        con = dict(zip(names, (float(v) for v in vals)))
        data = np.frombuffer(raw, "<f8", offset=16 * words).reshape(-1, words)
        self.cols = []
        for off, ncf, niv in cols:
            c = data[:, off - 1:off - 1 + 3 * ncf * niv].reshape(len(data), niv, 3, ncf)
            self.cols.append(torch.tensor(c.copy(), device="cuda"))
        e = self.emrat
        self.gm = [con["GMS"], con["GM1"], con["GM2"], con["GMB"] * e / (1 + e), con["GMB"] / (1 + e), con["GM4"],
                   con["GM5"], con["GM6"], con["GM7"], con["GM8"], con["GM9"]]
        raw = open(asteroids, "rb").read()
        count = int(struct.unpack_from("<d", raw, 1024 + 16)[0])
        self.ast = []
        for k in range(count):
            _, _, target, _, _, _, one, two = struct.unpack_from("<dd6i", raw, 1024 + 24 + 40 * k)
            seg = np.frombuffer(raw, "<f8", two - one + 1, 8 * (one - 1))
            init, intlen, rsize, nrec = seg[-4:]
            rec = seg[:int(rsize) * int(nrec)].reshape(int(nrec), int(rsize))[:, 2:]
            self.ast.append((init / 86400.0, intlen / 86400.0,
                             torch.tensor(rec.reshape(int(nrec), 3, -1).copy(), device="cuda")))
            self.gm.append(con["MA%04d" % (target - 2000000)])
        self.gm = torch.tensor(self.gm, dtype=torch.float64, device="cuda")
        self.j2, self.j3, self.j4, self.j2s = con["J2E"], con["J3E"], con["J4E"], con["J2SUN"]
        self.re, self.rs = con["RE"] / con["AU"], con["ASUN"] / con["AU"]
        self.oc2 = 1.0 / (con["CLIGHT"] * 86400.0 / con["AU"]) ** 2

    @staticmethod
    def _sums(coef, tau, rate):
        """sum c T, and its first and second derivatives by time; coef (..., 3, ncf)."""
        t, s, u = [torch.ones_like(tau), tau], [torch.zeros_like(tau), torch.ones_like(tau)], [torch.zeros_like(tau)] * 2
        for _ in range(coef.shape[-1] - 2):
            u.append(2 * tau * u[-1] + 4 * s[-1] - u[-2])
            s.append(2 * tau * s[-1] + 2 * t[-1] - s[-2])
            t.append(2 * tau * t[-1] - t[-2])
        return [(coef * torch.stack(w, -1)[..., None, :]).sum(-1) * rate ** k for k, w in enumerate((t, s, u))]

    def bodies(self, t):
        """Positions, velocities (AU, days) and accelerations of the bodies at
        times t of any shape: three tensors (27, *t.shape, 3); the asteroids'
        last two are NaN."""
        rel = (synth.JD_J2000 - self.beg) + t
        rec = torch.floor(rel / self.inc).long()
        frac = (rel - rec * self.inc) / self.inc
        col = []
        for c in self.cols:
            niv = c.shape[1]
            sub = torch.clamp((frac * niv).long(), 0, niv - 1)
            col.append(self._sums(c[rec, sub], 2 * (frac * niv - sub) - 1, 2.0 * niv / self.inc))
        out = []
        for k in range(3):
            emb, lun = col[2][k], col[9][k]
            earth, moon = emb - lun / (1 + self.emrat), emb + lun * (self.emrat / (1 + self.emrat))
            pl = [col[10][k], col[0][k], col[1][k], earth, moon] + [col[j][k] for j in range(3, 9)]
            out.append([p / self.au for p in pl])
        nan = torch.full_like(out[0][0], math.nan)
        for init, length, c in self.ast:
            b = torch.clamp(((t - init) / length).long(), 0, len(c) - 1)
            z = 2 * ((t - init) - b * length) / length - 1
            out[0].append(self._sums(c[b], z, 1.0)[0] / 149597870.7 + out[0][0])
            out[1].append(nan)
            out[2].append(nan)
        return [torch.stack(o) for o in out]

    def table(self, t):
        """What accel() needs of the bodies at times t: positions, the Sun's
        velocity, its acceleration by the planets and their potential there."""
        p, v, _ = self.bodies(t)
        d = p[0] - p[1:11]
        gm = self.gm[1:11].reshape(-1, *[1] * (d.dim() - 2))
        r = d.norm(dim=-1)
        return p, v[0], -((gm / r ** 3)[..., None] * d).sum(0), (gm / r).sum(0)

    def accel(self, tab, x, v, params):
        """The force model (its default terms) at x, v of shape (..., 3)."""
        pos, sun_v, sun_a, sun_u = tab
        d = x - pos
        r = torch.sqrt((d * d).sum(-1))
        gm = self.gm.reshape(-1, *[1] * (d.dim() - 2))
        dot = lambda a, b: (a * b).sum(-1, keepdim=True)  # noqa: E731
        # relativity: Einstein-Infeld-Hoffmann with the Sun as the source
        ds, rs = d[0], r[0][..., None]
        gs, oc2 = self.gm[0], self.oc2
        pre = gs / rs ** 3
        vs, us = sun_v, sun_u[..., None]
        factor = oc2 * (-4 * (gm / r)[:11].sum(0)[..., None] - us + dot(v, v) + 2 * dot(vs, vs) - 4 * dot(v, vs)
                        - 1.5 * (dot(ds, vs) / rs) ** 2 - 0.5 * dot(ds, sun_a))
        acc = -pre * factor * ds + oc2 * pre * dot(ds, 4 * v - 3 * vs) * (v - vs) + 3.5 * oc2 * gs / rs * sun_a
        # zonal harmonics of the Earth (pole along z) and of the Sun
        de, re = d[3], r[3][..., None]
        z = de[..., 2:]
        c2 = (z / re) ** 2
        k2 = 1.5 * self.gm[3] * self.j2 * self.re ** 2 / re ** 5
        k3 = 2.5 * self.gm[3] * self.j3 * self.re ** 3 / re ** 5
        k4 = 0.625 * self.gm[3] * self.j4 * self.re ** 4 / re ** 7
        pole = torch.tensor([0.0, 0.0, 1.0], dtype=torch.float64, device="cuda")
        acc = acc + (k2 * (5 * c2 - 1) - k3 * z / re ** 2 * (3 - 7 * c2) + k4 * (63 * c2 * c2 - 42 * c2 + 3)) * de
        acc = acc + (-2 * k2 * z - k3 * (3 * c2 - 0.6) + k4 * (12 - 28 * c2) * z) * pole
        ra, dec = math.radians(286.13), math.radians(63.87)
        pole = torch.tensor([math.cos(ra) * math.cos(dec), math.sin(ra) * math.cos(dec), math.sin(dec)],
                            dtype=torch.float64, device="cuda")
        z = (ds * pole).sum(-1, keepdim=True)
        k2 = 1.5 * gs * self.j2s * self.rs ** 2 / rs ** 5
        acc = acc + k2 * ((5 * (z / rs) ** 2 - 1) * ds - 2 * z * pole)
        # non-gravitational: radial, transverse and normal, 1 / r^2
        if params is not None:
            h = torch.linalg.cross(ds, v - vs)
            tr = torch.linalg.cross(h, ds)
            unit = lambda a: a / torch.sqrt(dot(a, a))  # noqa: E731
            acc = acc + (params[..., 0:1] * unit(ds) + params[..., 1:2] * unit(tr) + params[..., 2:3] * unit(h)) / rs ** 2
        return acc - ((gm / r ** 3)[..., None] * d).sum(0)

    def integrate(self, x, v, span, params, steps, outs):
        """x, v after span (one per particle) in equal steps of the eight-stage
        Gauss-Legendre collocation; outs: every so many steps the state is
        listed too (0: never)."""
        c, w = np.polynomial.legendre.leggauss(8)
        c = 0.5 * (c + 1)
        vander = np.vander(c, 8, increasing=True)
        a = (np.vander(c, 9, increasing=True)[:, 1:] / np.arange(1, 9)) @ np.linalg.inv(vander)
        a, b, c = (_gpu(q) for q in (a, 0.5 * w, c))
        a2, b2 = a @ a, b @ a
        h = span / steps
        same = bool((h == h[0]).all())
        hs = (h[:1] if same else h)
        got, acc = [], None
        for k in range(steps):
            tab = self.table(T0 + k * hs + c[:, None] * hs)
            if acc is None:
                acc = self.accel(self.table(T0 + 0 * hs), x, v, params).expand(8, -1, -1).clone()
            hh = h[:, None]
            for _ in range(40):
                xs = x + (c[:, None, None] * hh) * v + hh * hh * torch.einsum("ij,jnk->ink", a2, acc)
                vs = v + hh * torch.einsum("ij,jnk->ink", a, acc)
                new = self.accel(tab, xs, vs, params)
                off = float(((new - acc).norm(dim=-1) / new.norm(dim=-1)).max())
                acc = new
                if off < 3e-15:
                    break
            x = x + hh * v + hh * hh * torch.einsum("j,jnk->nk", b2, acc)
            v = v + hh * torch.einsum("j,jnk->nk", b, acc)
            if outs and (k + 1) % outs == 0:
                got.append(torch.cat([x, v], -1))
        return x, v, got


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    x = _inputs(case, seed)
    e = _World.get().plain()
    if kind == "bodies":
        p, v, a = e.bodies(_gpu(x["t"]))
        gm = e.gm[:, None, None].expand(-1, n, 1)
        return torch.cat([gm, p, v, a], -1).transpose(0, 1)
    state, params = _gpu(x["state"]), _gpu(x.get("params"))
    if kind in ("forces", "shared"):
        tab = e.table(_gpu(x["t"]))
        pos, vel = state[:, :3], state[:, 3:]
        acc = e.accel(tab, pos, vel, params)
        if kind == "shared":
            return acc
        if not case["var"]:
            return {"acc": acc}
        # derivatives along the variational states by complex steps
        var, h, cols = _gpu(x["var"]), 1e-30, []
        for k in range(6):
            z = torch.complex(state, h * var[:, k])
            cols.append(e.accel(tab, z[:, :3], z[:, 3:], params).imag / h)
        return {"acc": acc, "var_acc": torch.stack(cols, 1)}
    per_step = 4.0 if case["pop"] == "mba" else 1.25
    steps = max(8, int(math.ceil(case["days"] / per_step)))
    if float(n) * steps > 1.5e6:
        return None                   # too long for plain arithmetic
    span, outs = _gpu(x["span"]) if "span" in x else torch.full((n,), case["days"], dtype=torch.float64, device="cuda"), 0
    if case.get("every"):
        outs = max(1, int(math.ceil(case["every"] / per_step)))
        steps = outs * len(x["out"])
    px, pv, got = e.integrate(state[:, :3].clone(), state[:, 3:].clone(), span, params, steps, outs)
    end = torch.cat([px, pv], -1)
    if kind == "dropin":
        return end if not case["var"] else None
    out = {"state": end, "status": torch.zeros(n, dtype=torch.int32)}
    if outs:
        out["dense"] = torch.stack(got, 1).reshape(-1, 6)
    return out
