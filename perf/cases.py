"""Timed cases of the engine: what its users run, over the sizes they run it at.

A case is a dict of plain values.  Its "kind" names the call sequence:

  group    Engine.run(steps, meas_every), cancel_vcom, and the state back to
           page-locked host arrays: one group of md.F's step loop (md.F:87-101)
           as the Python driver makes it
  newton   one Engine.newton and the new positions and velocities on the host:
           the Fortran shim's step, one call at a time
  accel    one measuring Engine.accel of positions that the host has just set,
           and the accelerations on the host (the reference's accel(.true.))
  batch    Batch.run(steps, meas_every) of an ensemble of small boxes, and
           every box's state on the host
  gofr     Engine.gofr_counts, the pair histogram of g(r)
  noalloc  accel_noalloc on device arrays that the caller owns

"sim" and the physical constants follow yukawamd_b200.configs: ions at its
density with r_c = min(L/2, 10 lambda), nucleons at 0.05 fm^-3 with the
automatic nuclear cutoff and an uncut p-p Coulomb term.  Positions are those
of a dense liquid (a jittered, randomly occupied and randomly ordered lattice:
no overlaps, short-range order), not the uniform random start that a run
leaves behind after its first steps.

FP64 boxes return 64-bit values.  The mixed form computes its pair terms in 32
bits, so its forces, energies and the trajectories that they drive are worth 32
bits, and a program that asks for that form takes them as 32-bit values.
"""
import math

import numpy as np
import torch

from yukawamd_b200 import abi, configs
from yukawamd_b200.engine import Batch, Engine, accel_noalloc

PRECISION = {"fp64": abi.YK_PREC_FP64, "mixed": abi.YK_PREC_MIXED}

# Flops of one pair, force-only and measuring (sums over unique pairs).
ION_FLOPS = {False: 30, True: 47}
NUCLEAR_FLOPS = {False: 21, True: 38}
COULOMB_FLOPS = {False: 28, True: 45}


def listed():
    return [
        # The shortest call of a step-at-a-time driver: a small box that a
        # desktop run would use, one newton per call.
        dict(name="newton-ion-500-fp64", kind="newton", sim="pure", n=500, prec="fp64", kappa=1.0, gamma=175.0,
             integrator=2),
        # The smallest benchmark configuration in both forms: a warm-up group
        # of 100 steps of the pure-ion OCP.
        dict(name="group-ion-4096-fp64", kind="group", sim="pure", n=4096, prec="fp64", kappa=1.0, gamma=175.0,
             steps=100, meas=0, integrator=2),
        dict(name="group-ion-4096-mixed", kind="group", sim="pure", n=4096, prec="mixed", kappa=1.0, gamma=175.0,
             steps=100, meas=0, integrator=2),
        # The headline configuration in both forms: production steps of the
        # 55,296-ion mixture, measuring every 10th.
        dict(name="group-mix-55296-fp64", kind="group", sim="mix", n=55296, prec="fp64", kappa=0.5, gamma=150.0,
             steps=20, meas=10, integrator=2),
        dict(name="group-mix-55296-mixed", kind="group", sim="mix", n=55296, prec="mixed", kappa=0.5, gamma=150.0,
             steps=20, meas=10, integrator=2),
        # Nucleon matter in both forms, the reference's nuclear-pasta runs.
        dict(name="group-nn-51200-fp64", kind="group", sim="nucleon", n=51200, prec="fp64", steps=10, meas=5,
             integrator=2),
        dict(name="group-nn-51200-mixed", kind="group", sim="nucleon", n=51200, prec="mixed", steps=10, meas=5,
             integrator=2),
        # A measuring force call of a strained (rectangular) box with an odd
        # particle count and stronger screening.
        dict(name="accel-mix-12345-fp64", kind="accel", sim="mix", n=12345, prec="fp64", kappa=1.3, gamma=90.0,
             aspect=1.2),
        # The largest box that is served: one force call of 131,072 ions.
        dict(name="accel-ion-131072-mixed", kind="accel", sim="pure", n=131072, prec="mixed", kappa=1.0,
             gamma=120.0, aspect=1.0),
        # An ensemble of uneven replicas in one batch, as the serving groups
        # and the replica studies run it.
        dict(name="batch-24-mixed", kind="batch", count=24, nmin=1000, nmax=20000, prec="mixed", steps=50, meas=10),
        # g(r) of one configuration of a medium box, 500 bins.
        dict(name="gofr-ion-27000", kind="gofr", sim="pure", n=27000, nbin=500, kappa=1.0, gamma=175.0),
        # Forces inside an application that owns the device memory.
        dict(name="noalloc-mix-2000-fp64", kind="noalloc", sim="mix", n=2000, prec="fp64", kappa=0.8, gamma=120.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["group", "group", "group", "accel", "accel", "newton", "batch", "gofr", "noalloc"])
    prec = rng.choice(["fp64", "mixed"])
    kappa, gamma = round(rng.uniform(0.5, 2.0), 3), round(rng.uniform(50.0, 250.0), 1)
    sim = rng.choice(["pure", "mix", "nucleon"])
    ions = dict(kappa=kappa, gamma=gamma) if sim != "nucleon" else {}
    if kind == "group":
        n = _log_int(rng, 512, 55000)
        # no costlier than the largest listed group
        most = max(4, int(20 * (55000.0 / n) ** 2))
        # (nucleons take few steps: at dt = 2 fm/c their collisions amplify a
        # rounding error a hundredfold within 20)
        steps = min(rng.choice([12, 20, 40, 100] if ions else [4, 8, 12]), most)
        return dict(kind=kind, sim=sim, n=n, prec=prec, steps=steps, meas=rng.choice([0, 4, 10]),
                    integrator=rng.choice([1, 2, 2]), **ions)
    if kind == "accel":
        return dict(kind=kind, sim=sim, n=_log_int(rng, 512, 131072), prec=prec,
                    aspect=rng.choice([1.0, round(rng.uniform(0.8, 1.4), 3)]), **ions)
    if kind == "newton":
        return dict(kind=kind, sim=sim, n=_log_int(rng, 100, 8192), prec=prec, integrator=2, **ions)
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(4, 24), nmin=rng.randint(500, 1000), nmax=rng.randint(2000, 20000),
                    prec=prec, steps=rng.choice([10, 50]), meas=rng.choice([0, 10]))
    if kind == "gofr":
        return dict(kind=kind, sim="pure", n=_log_int(rng, 512, 40000), nbin=rng.choice([100, 500, 2000]),
                    kappa=kappa, gamma=gamma)
    return dict(kind=kind, sim=sim, n=_log_int(rng, 100, 4096), prec=prec, **ions)


# ---- inputs ---------------------------------------------------------------

def _liquid(rng, n, xl):
    """n positions of a dense liquid in the box xl: cells of a cubic lattice,
    occupied at random and in random order, jittered by a clipped normal."""
    m = math.ceil(n ** (1.0 / 3.0) - 1e-9)
    cell = rng.permutation(m ** 3)[:n]
    idx = np.stack([cell // (m * m), cell // m % m, cell % m], axis=1)
    jit = np.clip(0.14 * rng.standard_normal((n, 3)), -0.4, 0.4)
    return np.ascontiguousarray((idx + 0.5 + jit) / m * np.asarray(xl)).reshape(-1)


def _workload(case, seed):
    """The case's box: parameters and velocities of yukawamd_b200.configs,
    liquid positions, and the box strained to its aspect ratio."""
    n = case["n"]
    if case["sim"] == "pure":
        w = configs.pure_ion(n, 8, 16, case["kappa"], case["gamma"], seed)
    elif case["sim"] == "mix":
        w = configs.ion_mixture(n, [6, 8, 26], [0.2, 0.7, 0.1], case["kappa"], case["gamma"], seed)
    else:
        w = configs.nucleon(n, 0.4, 0.05, 1.0, 10.0, 2.0, seed)
    aspect = case.get("aspect", 1.0)
    if aspect != 1.0:
        edge = w.params["xl"][0]
        w.params["xl"] = [edge / math.sqrt(aspect), edge / math.sqrt(aspect), edge * aspect]
        w.params["rccut"] = min(w.params["rccut"], min(w.params["xl"]) / 2.0) if case["sim"] != "nucleon" \
            else w.params["rccut"]
    w.x = _liquid(np.random.default_rng([seed, 7]), n, w.params["xl"])
    w.params["precision"] = PRECISION[case.get("prec", "fp64")]
    w.params["integrator"] = case.get("integrator", 2)
    return w


def _replicas(case):
    """The batch's boxes: pure-ion and mixture replicas, their sizes spread over
    the logarithm of [nmin, nmax] and kappa and Gamma over their ranges, in an
    order that mixes all three."""
    count, out = case["count"], []
    for r in range(count):
        q = ((7 * r) % count + 0.5) / count
        n = int(round(case["nmin"] * (case["nmax"] / case["nmin"]) ** q))
        out.append(dict(sim="pure" if r % 2 else "mix", n=n, prec=case["prec"], kappa=0.5 + 1.5 * (0.618 * r % 1.0),
                        gamma=50.0 + 200.0 * (0.414 * r % 1.0)))
    return out


def _boxes(case, seed):
    rng = np.random.default_rng([seed, 11])
    return [_workload(one, int(rng.integers(1 << 30))) for one in _replicas(case)]


def _pinned(count):
    return torch.empty(count, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        batch = Batch(_boxes(case, seed), mix_mode=abi.YK_MIX_FIXED)
        batch.accel(True)                          # md.F:69
        return dict(case=case, batch=batch)
    w = _workload(case, seed)
    if kind == "noalloc":
        dev = torch.device("cuda", 0)
        up = [torch.from_numpy(t).to(dev) for t in (w.x, w.zii, w.aii)]
        a = torch.zeros(3 * (w.n + 3), dtype=torch.float64, device=dev)
        return dict(case=case, params=w.yk_params(), n=w.n, up=up, a=a)
    state = dict(case=case, engine=Engine(w), out=[_pinned(3 * w.n) for _ in range(3)])
    if kind in ("group", "newton"):
        state["engine"].accel(True, fetch_a=False)  # md.F:69
    if kind == "accel":
        state["x"] = _pinned(3 * w.n)
        state["x"][:] = w.x
    return state


# ---- one pass ------------------------------------------------------------

def _values(case, v):
    """Results in the precision that the form computes them in."""
    v = np.asarray(v)
    return v.astype(np.float32) if case.get("prec") == "mixed" else v


def _scalars(case, s):
    return {"ev": _values(case, s.ev), "px": _values(case, s.px), "ek": _values(case, s.ek),
            "pp": _values(case, s.pp[:])}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        b = state["batch"]
        series, _ = b.run(case["steps"], case["meas"], series=case["meas"] > 0)
        states = [b.get_state(r) for r in range(b.nrep)]
        out = {"x": _values(case, np.concatenate([s[0] for s in states])),
               "v": _values(case, np.concatenate([s[1] for s in states]))}
        if case["meas"]:
            last = case["steps"] // case["meas"] * case["meas"] - 1
            out["ev"] = _values(case, [series[last * b.nrep + r].ev for r in range(b.nrep)])
        return out
    if kind == "noalloc":
        x, zii, aii = state["up"]
        s = accel_noalloc(state["params"], state["n"], x.data_ptr(), zii.data_ptr(), aii.data_ptr(), True,
                          state["a"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        a = state["a"][:3 * state["n"]]
        return {"a": a.float() if case["prec"] == "mixed" else a, "ev": _values(case, s.ev),
                "px": _values(case, s.px)}
    e = state["engine"]
    if kind == "gofr":
        return {"counts": e.gofr_counts(case["nbin"]).astype(np.int64)}
    x, v, a = state["out"]
    if kind == "accel":
        e.set_state(x=state["x"])
        s = e.accel(True, fetch_a=False)
        e.get_into(a=a)
        return {"a": _values(case, a), "ev": _values(case, s.ev), "px": _values(case, s.px),
                "pp": _values(case, s.pp[:])}
    if kind == "newton":
        s = e.newton(True)
        e.get_into(x=x, v=v)
        return {"x": _values(case, x), "v": _values(case, v), **_scalars(case, s)}
    series = e.run(case["steps"], case["meas"], series=case["meas"] > 0)
    e.cancel_vcom()
    e.get_into(x=x, v=v, a=a)
    out = {"x": _values(case, x), "v": _values(case, v), "a": _values(case, a)}
    if case["meas"]:
        last = case["steps"] // case["meas"] * case["meas"] - 1
        if last >= 0:
            out.update(_scalars(case, series[last]))
    return out


# ---- what a pass cannot do without ------------------------------------------

def _pair_flops(case, meas):
    """Flops of the pairs inside the cutoffs of one force call."""
    n = case["n"]
    if case["sim"] == "nucleon":
        near = 4.0 / 3.0 * math.pi * configs.rncut_auto() ** 3 * 0.05
        np_ = 0.4 * n
        return 0.5 * n * min(near, n - 1) * NUCLEAR_FLOPS[meas] + 0.5 * np_ * (np_ - 1) * COULOMB_FLOPS[meas]
    length = (n / configs.ION_DENSITY) ** (1.0 / 3.0)
    a_ws = (3.0 / (4.0 * math.pi * configs.ION_DENSITY)) ** (1.0 / 3.0)
    rc = min(0.5 * length, 10.0 * a_ws / case["kappa"])
    return 0.5 * n * min(4.0 / 3.0 * math.pi * rc ** 3 * configs.ION_DENSITY, n - 1) * ION_FLOPS[meas]


def work(case):
    kind = case["kind"]
    if kind == "batch":
        boxes, measured = _replicas(case), case["steps"] // case["meas"] if case["meas"] else 0
        return dict(bytes=96.0 * sum(one["n"] for one in boxes),
                    flops=sum((case["steps"] - measured) * _pair_flops(one, False) +
                              measured * _pair_flops(one, True) for one in boxes))
    n = case["n"]
    if kind == "gofr":
        return dict(bytes=24.0 * n + 8.0 * case["nbin"], flops=0.5 * n * (n - 1) * 15.0)
    if kind == "group":
        measured = case["steps"] // case["meas"] if case["meas"] else 0
        return dict(bytes=120.0 * n, flops=(case["steps"] - measured) * _pair_flops(case, False) +
                    measured * _pair_flops(case, True))
    return dict(bytes=(88.0 if kind == "newton" else 64.0) * n, flops=_pair_flops(case, True))


# ---- the same in plain 64-bit torch -------------------------------------------

class _Exact:
    """The reference's algorithm on all ordered pairs, row blocks at a time."""

    def __init__(self, p, x, v, zii, aii, dev):
        self.p, self.dev = p, dev
        self.n = len(zii)
        self.x = torch.from_numpy(np.array(x)).to(dev).view(-1, 3)
        self.v = torch.from_numpy(np.array(v)).to(dev).view(-1, 3)
        self.z = torch.from_numpy(np.array(zii)).to(dev)
        self.m = torch.from_numpy(np.array(aii)).to(dev)
        self.xl = torch.tensor(list(p.xl), dtype=torch.float64, device=dev)

    def force(self, meas):
        p, n, x, z = self.p, self.n, self.x, self.z
        ion = p.sim_type != abi.YK_SIM_NUCLEON
        pure = p.sim_type == abi.YK_SIM_PURE_ION
        diag = math.sqrt(sum(t * t for t in p.xl)) / 2.0
        cut = math.exp(-p.xmuc * p.rccut) / p.rccut if p.rccut <= diag else 0.0
        f = torch.empty_like(x)
        sums = torch.zeros(8, dtype=torch.float64, device=self.dev)       # U, W, xx, xy, xz, yy, yz, zz
        rows = max(1, min(n, (1 << 25) // n))
        for i0 in range(0, n, rows):
            xi = x[i0:i0 + rows]
            d = []
            for k in range(3):
                t = xi[:, k, None] - x[None, :, k]
                half = 0.5 * p.xl[k]
                d.append(torch.where(t > half, t - p.xl[k], torch.where(t < -half, t + p.xl[k], t)))
            r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
            own = torch.arange(xi.shape[0], device=self.dev)
            r2[own, i0 + own] = math.inf
            fs = torch.zeros_like(r2)
            u = torch.zeros_like(r2)
            if ion:
                on = r2 <= p.rccut * p.rccut
                r = torch.where(on, r2, 1.0).sqrt()
                er = torch.exp(-p.xmuc * r) / r
                fs = torch.where(on, (1.0 + p.xmuc * r) * er / (r * r), 0.0)
                u = torch.where(on, er - cut, 0.0) if meas else u
                if not pure:
                    fs *= z[None, :]
                    u = u * z[None, :]
            else:
                if p.nuclear_on:
                    on = r2 <= p.rncut * p.rncut
                    e = torch.where(on, torch.exp(-torch.where(on, r2, 0.0) / (2.0 * p.xpacket)), 0.0)
                    b = torch.where(z[i0:i0 + rows, None] == z[None, :], p.bb + p.cc, p.bb - p.cc)
                    fs += (2.0 * p.aa * e + b) * e / p.xpacket
                    u += (p.aa * e + b) * e
                if p.coulomb_on:
                    on = (r2 <= p.rccut * p.rccut) & torch.isfinite(r2) & (z[i0:i0 + rows, None] == 1.0) & \
                        (z[None, :] == 1.0)
                    r = torch.where(on, r2, 1.0).sqrt()
                    er = p.vc * torch.exp(-p.xmuc * r) / r
                    fs += torch.where(on, (1.0 + p.xmuc * r) * er / (r * r), 0.0)
                    u += torch.where(on, er - p.vc * cut, 0.0)
            g = [fs * t for t in d]
            for k in range(3):
                f[i0:i0 + rows, k] = g[k].sum(1)
            if meas:
                zi = z[i0:i0 + rows] if ion and not pure else torch.ones(xi.shape[0], dtype=torch.float64,
                                                                         device=self.dev)
                rowsum = [u.sum(1), (g[0] * d[0] + g[1] * d[1] + g[2] * d[2]).sum(1)] + \
                    [(d[a] * g[b]).sum(1) for a, b in ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))]
                sums += 0.5 * torch.stack([(zi * t).sum() for t in rowsum])
        if pure:
            coef = p.frp * p.zi * p.zi * p.vc
            self.a = coef * f / (p.ai * p.xmass)
        elif ion:
            coef = p.frp * p.vc
            fold = z.clone()
            if p.mix_mode == abi.YK_MIX_COMPAT:
                fold[n - 1] = 1.0                          # int_ion_mix.f:158,201
            self.a = coef * f * fold[:, None] / (self.m * p.xmass)[:, None]
        else:
            coef = 1.0
            self.a = f / p.xmass
        if not meas:
            return None
        s = (coef * sums).tolist()
        pp = np.array([s[2], s[3], s[4], s[3], s[5], s[6], s[4], s[6], s[7]])
        return dict(ev=s[0] / n, px=p.rho * (p.kT + s[1] / (3.0 * n)), pp=pp)

    def step(self, meas):
        p, dt = self.p, self.p.dt
        x = self.x + self.v * dt + 0.5 * dt * dt * self.a
        x = torch.where(x < 0.0, x + self.xl, x)
        self.x = torch.where(x > self.xl, x - self.xl, x)
        half = self.v + 0.5 * dt * self.a
        s = self.force(meas)
        self.v = half + 0.5 * dt * self.a
        if meas:
            kin = (p.xmass * (self.m[:, None, None] * self.v[:, :, None] * self.v[:, None, :]).sum(0)).cpu().numpy()
            s["ek"] = 0.5 * float(np.trace(kin)) / self.n
            s["pp"] = (s["pp"] + kin.reshape(-1)) / (p.xl[0] * p.xl[1] * p.xl[2])
        return s

    def cancel_vcom(self):
        p = self.p
        v = self.v - (self.m[:, None] * self.v).sum(0) / self.m.sum()
        eka = 0.5 * p.xmass * float((self.m * (v * v).sum(1)).sum()) / self.n
        self.v = v / math.sqrt(eka / (1.5 * p.kT))


def _exact_box(w, mix_mode=abi.YK_MIX_COMPAT):
    dev = torch.device("cuda", 0) if torch.cuda.is_available() else torch.device("cpu")
    return _Exact(w.yk_params(mix_mode=mix_mode), w.x, w.v, w.zii, w.aii, dev)


def _host(t):
    return t.reshape(-1).cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "gofr":
        return None                                        # whole numbers
    if kind == "batch":
        xs, vs, evs = [], [], []
        for w in _boxes(case, seed):
            e = _exact_box(w, abi.YK_MIX_FIXED)
            e.force(False)
            ev = 0.0
            for s in range(1, case["steps"] + 1):
                meas = case["meas"] > 0 and s % case["meas"] == 0
                got = e.step(meas)
                ev = got["ev"] if meas else ev
            xs.append(_host(e.x))
            vs.append(_host(e.v))
            evs.append(ev)
        out = {"x": np.concatenate(xs), "v": np.concatenate(vs)}
        if case["meas"]:
            out["ev"] = np.array(evs)
        return out
    e = _exact_box(_workload(case, seed))
    s = e.force(True)
    if kind in ("accel", "noalloc"):
        out = {"a": _host(e.a), "ev": np.array(s["ev"]), "px": np.array(s["px"])}
        if kind == "accel":
            out["pp"] = s["pp"]
        return out
    last = None
    steps = 1 if kind == "newton" else case["steps"]
    for k in range(1, steps + 1):
        meas = kind == "newton" or (case["meas"] > 0 and k % case["meas"] == 0)
        got = e.step(meas)
        last = got if meas else last
    if kind == "group":
        e.cancel_vcom()
    out = {"x": _host(e.x), "v": _host(e.v)}
    if kind == "group":
        out["a"] = _host(e.a)
    if last:
        out.update({k: np.array(v) for k, v in last.items()})
    return out
