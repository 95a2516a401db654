"""The work that users of this framework have it do, as cases that can be timed
and checked: integrating planetesimal disks through the pp_disk / integrator
seam, the diagnostics at an output time, the gravity of device arrays, and the
training step of the step-size network.

A case is a dict of plain values.  `listed()` gives the fixed ones, `draw(rng)`
one more of the same ranges, `prepare` builds what a user's program holds
before the call, `run` makes one pass through the public entry points, `work`
says what a pass cannot do without and `exact` gives a pass's result in 64 bits
with torch alone.

Units: AU, solar masses, code time (1/k days).
"""
import math
from types import SimpleNamespace

import numpy as np
import torch

import __graft_entry__

rg = __graft_entry__.load_package()

K = 0.01720209895                   # Gauss's constant: code time = days * K
EARTH = 1.0 / 3.3294605e5           # M_sun
RHO = 2.0 * (1.495978707e13 ** 3) / 1.98911e33   # 2 g/cm^3 in M_sun / AU^3
CADENCE = 0.25 * K                  # the adaptive runs' output interval: four snapshots a day
CUBE_DT = 1.0e-3


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _disk(name, kind, n_pp, n_pl, **kw):
    c = {"name": name, "kind": kind, "field": "disk", "n_pp": n_pp, "n_pl": n_pl, "n_tp": 0, "systems": 1,
         "integrator": "rkf78", "adaptive": True, "precision": "mixed", "gas": False, "tries": 1}
    c.update(kw)
    return c


def listed():
    return [
        # one integrator step of a small disk, state in and state out: the call of an
        # interactive program, or of one that couples the disk to other physics every
        # step; launches, synchronisations and transfers are its cost
        _disk("step_261", "step", 4, 256),
        # red's CPU-sized run: 2053 bodies, fixed-step RK4, many steps at a time
        _disk("rk4_2053", "run", 4, 2048, integrator="rk4", adaptive=False, tries=100),
        # the headline workload: a 16384-body disk, adaptive RKF7(8), collisions on
        _disk("disk_16384", "run", 16, 16367, tries=40),
        # the same disk in FP64 arithmetic, the mode a user checks MIXED against
        _disk("disk_16384_fp64", "run", 16, 16367, precision="fp64", tries=10),
        # red's own arithmetic bit for bit, the mode that reproduces red's runs
        _disk("exact_4100", "run", 8, 4091, precision="fp64_exact", tries=4),
        # the largest single disk, with gas drag
        _disk("gas_65536", "run", 32, 65503, gas=True, tries=10),
        # a parameter study: 512 disks of 128 to 4096 bodies side by side
        _disk("ensemble_512", "run", 0, 0, systems=512, n_min=128, n_max=4096, tries=4),
        # every pair of 16384 bodies interacting (a disk of protoplanets)
        _disk("allpairs_16384", "run", 16, 16367, field="allpairs", tries=4),
        # red's benchmark cube at its largest size, FP32 pair terms, RK4
        _disk("cube_65536_fp32", "run", 0, 65536, field="cube", integrator="rk4", adaptive=False, precision="fp32",
              tries=2),
        # gravity of arrays that live on the device, for a program with its own
        # integrator: an odd number of bodies
        _disk("accel_20011", "accel", 12, 19998),
        # what a run prints at an output time: integrals, energy over the interacting
        # pairs, the overlapping pairs at five times the radii, the state
        _disk("output_16384", "output", 16, 16367),
        # one training step of the step-size network on the trainer's batch
        {"name": "train_2048", "kind": "train", "rows": 2048},
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    what = rng.choice(["step", "disk", "disk", "disk", "gas", "ensemble", "allpairs", "cube", "accel", "output",
                       "train"])
    scheme = rng.choice(["rkf78", "rkf78", "rkf78", "rk4", "rk2", "euler"])
    flow = {"integrator": scheme, "adaptive": scheme == "rkf78" or (scheme == "rk4" and rng.random() < 0.5)}
    mode = rng.choice(["mixed", "mixed", "mixed", "fp32", "fp64"])
    if what == "train":
        return _unnamed({"kind": "train", "rows": logint(48, 65536)})
    if what == "step":
        return _unnamed(_disk("", "step", rng.randint(2, 16), logint(64, 16384), systems=rng.choice([1, 1, 1, 4, 16]),
                              **flow, precision=mode))
    if what == "disk":
        if rng.random() < 0.2:
            return _unnamed(_disk("", "run", rng.randint(2, 8), logint(128, 4096), **flow, precision="fp64_exact",
                                  tries=rng.randint(2, 4)))
        n_pl = logint(128, 65536)
        n_tp = rng.choice([0, 0, 0, rng.randint(1, 200)])
        return _unnamed(_disk("", "run", rng.randint(2, 32), n_pl, n_tp=n_tp, **flow, precision=mode,
                              tries=rng.randint(5, 20)))
    if what == "gas":
        return _unnamed(_disk("", "run", rng.randint(2, 32), logint(1024, 65503), gas=True, **flow, precision="mixed",
                              tries=rng.randint(4, 10)))
    if what == "ensemble":
        n_max = logint(256, 4096)
        return _unnamed(_disk("", "run", 0, 0, systems=logint(8, 512), n_min=rng.randint(100, 128), n_max=n_max,
                              **flow, precision=rng.choice(["mixed", "mixed", "fp32"]), tries=rng.randint(2, 4)))
    if what == "allpairs":
        return _unnamed(_disk("", "run", rng.randint(2, 16), logint(512, 16367), field="allpairs", **flow,
                              precision=rng.choice(["mixed", "mixed", "fp32"]), tries=rng.randint(2, 4)))
    if what == "cube":
        return _unnamed(_disk("", "run", 0, logint(1024, 50000), field="cube", integrator="rk4", adaptive=False,
                              precision=rng.choice(["fp32", "mixed"]), tries=rng.randint(1, 2)))
    if what == "accel":
        if rng.random() < 0.4:
            return _unnamed(_disk("", "accel", rng.randint(2, 16), logint(256, 16367), field="allpairs",
                                  precision=rng.choice(["mixed", "fp32"])))
        return _unnamed(_disk("", "accel", rng.randint(2, 32), logint(128, 32000), precision=mode))
    return _unnamed(_disk("", "output", rng.randint(2, 32), logint(1024, 32768)))


def _unnamed(c):
    c.pop("name", None)
    return c


# ---------------------------------------------------------------------------
# inputs (from the seed alone; plain numpy)
# ---------------------------------------------------------------------------
def _kepler(rng, a, sigma_e, sigma_i, m):
    """Positions and velocities of bodies on Rayleigh-distributed Kepler orbits of a star of unit mass."""
    n = len(a)
    e = np.minimum(rng.rayleigh(1.0, n) * sigma_e, 0.9)
    inc = rng.rayleigh(1.0, n) * sigma_i
    peri, node, mean = (rng.uniform(0.0, 2.0 * math.pi, n) for _ in range(3))
    E = mean + e * np.sin(mean)
    for _ in range(8):
        E -= (E - e * np.sin(E) - mean) / (1.0 - e * np.cos(E))
    q = np.sqrt(1.0 - e * e)
    X, Y = a * (np.cos(E) - e), a * q * np.sin(E)
    f = np.sqrt((1.0 + m) / a) / (1.0 - e * np.cos(E))
    VX, VY = -f * np.sin(E), f * q * np.cos(E)
    cw, sw, cO, sO, ci, si = np.cos(peri), np.sin(peri), np.cos(node), np.sin(node), np.cos(inc), np.sin(inc)
    P = np.stack([cw * cO - sw * sO * ci, cw * sO + sw * cO * ci, sw * si], axis=1)
    Q = np.stack([-sw * cO - cw * sO * ci, -sw * sO + cw * cO * ci, cw * si], axis=1)
    return X[:, None] * P + Y[:, None] * Q, VX[:, None] * P + VY[:, None] * Q


def _bodies(case, seed):
    """All systems' bodies one after the other: r, v (n x 3), mass, radius, cd, type, and the counts per system."""
    rng = np.random.default_rng(int(seed))
    if case["field"] == "cube":
        n = case["n_pl"]
        r = rng.uniform(-50.0, 50.0, (n, 3))
        v = rng.normal(0.0, math.sqrt(0.2 * n / 50.0), (n, 3))
        one = np.ones(n)
        return SimpleNamespace(r=r, v=v, m=one, R=1e-3 * one, cd=0.0 * one, rho=one,
                               ty=np.full(n, rg.types.PROTOPLANET), counts=[(0, n, 0, 0)])
    if case["systems"] > 1 and "n_max" in case:
        sizes = np.random.default_rng(1000)              # the disks' sizes belong to the case, not to the seed
        counts = []
        for n in sizes.integers(case["n_min"], case["n_max"] + 1, case["systems"]):
            pp = int(sizes.integers(2, 9))
            counts.append((1, pp, int(n) - 1 - pp, 0))
    else:
        counts = [(1, case["n_pp"], case["n_pl"], case["n_tp"])] * case["systems"]
    wide = case["n_pp"] > 8
    n_pp = np.array([c[1] for c in counts])
    n_pl = np.array([c[2] for c in counts])
    n_tp = np.array([c[3] for c in counts])
    ns = 1 + n_pp + n_pl + n_tp
    off = np.concatenate([[0], np.cumsum(ns)])[:-1]
    sysof = np.repeat(np.arange(len(counts)), ns)
    k = np.arange(ns.sum()) - off[sysof]
    star = k == 0
    pp = (k >= 1) & (k <= n_pp[sysof])
    tp = k >= 1 + n_pp[sysof] + n_pl[sysof]
    m_pp = (0.05 if wide else 0.1) * EARTH
    h = (2.0 * m_pp / 3.0) ** (1.0 / 3.0)
    ratio = (1.0 + 5.0 * h) / (1.0 - 5.0 * h)           # 10 mutual Hill radii apart
    lo, hi = (0.5, 3.0) if wide else (0.7, 1.5)
    a = np.exp(rng.uniform(math.log(lo), math.log(hi), len(k))) if wide else rng.uniform(lo, hi, len(k))
    a[pp] = 0.5 * ratio ** (k[pp] - 1) if wide else 0.8 + 0.2 * (k[pp] - 1)
    m = np.zeros(len(k))
    if case["gas"]:                                     # radii log-uniform in 1 .. 100 km
        R = np.exp(rng.uniform(0.0, math.log(100.0), len(k))) / 1.495978707e8
        m = 4.0 / 3.0 * math.pi * R ** 3 * RHO
    else:
        m = EARTH / np.maximum(1, n_pl)[sysof]
    m[pp] = m_pp
    m[tp] = 0.0
    m[star] = 1.0
    R = np.cbrt(m / (4.0 / 3.0 * math.pi * RHO))
    R[star] = 1.0 / 215.094
    s = 0.02 if wide else 0.01
    r, v = _kepler(rng, a, s, 0.5 * s, m)
    r[star] = 0.0
    v[star] = 0.0
    w = m[:, None]
    M = np.add.reduceat(w, off)                          # each system to its barycentre
    r -= (np.add.reduceat(w * r, off) / M)[sysof]
    v -= (np.add.reduceat(w * v, off) / M)[sysof]
    ty = np.where(star, rg.types.STAR, np.where(pp, rg.types.PROTOPLANET, np.where(tp, rg.types.TESTPARTICLE,
                                                                                 rg.types.PLANETESIMAL)))
    if case["field"] == "allpairs":
        ty = np.where(star, rg.types.STAR, rg.types.PROTOPLANET)
        counts = [(1, c[1] + c[2], 0, 0) for c in counts]
    cd = np.where(case["gas"] & ~star & ~pp, 0.44, 0.0)
    if case["kind"] == "output":                         # a dozen planetesimals touch another one
        first = 1 + case["n_pp"]
        i = first + 2 * rng.choice(case["n_pl"] // 2 - 1, 12, replace=False)
        u = rng.normal(size=(12, 3))
        u /= np.linalg.norm(u, axis=1)[:, None]
        r[i + 1] = r[i] + u * (rng.uniform(0.5, 4.0, 12) * (R[i] + R[i + 1]))[:, None]
    return SimpleNamespace(r=r, v=v, m=m, R=R, cd=cd, rho=np.full(len(k), RHO), ty=ty, counts=counts)


def _gas():
    """The minimum-mass nebula's surface density (1700 g/cm^2 at 1 AU), h/r = 0.05, eta = 0.002."""
    keys = {"time_dependence": "constant", "eta_c": 0.002, "eta_p": 0.0, "rho_p": -2.5, "sch_c": 0.05, "sch_p": 1.0,
            "rho_c": 1700.0 / (math.sqrt(math.pi) * 0.05 * 1.495978707e13), "mmw": 2.3, "diameter": 3.0e-10,
            "alpha": 2.0e-3, "tau_c": 0.0, "tau_p": 0.0}
    return rg.ic.gas_params(keys)


def _var4(a):
    out = np.zeros(len(a), rg.types.VAR4)
    out["x"], out["y"], out["z"] = a[:, 0], a[:, 1], a[:, 2]
    return out


def _pinned(n, dtype, like=None):
    a = torch.zeros(n * dtype.itemsize, dtype=torch.uint8, pin_memory=True).numpy().view(dtype)
    if like is not None:
        a[:] = like
    return a


def _sim(case, b):
    """The handle a program keeps, and its page-locked state arrays."""
    p = np.zeros(len(b.m), rg.types.PARAM)
    p["mass"], p["radius"], p["density"], p["cd"] = b.m, b.R, b.rho, b.cd
    md = np.zeros(len(b.m), rg.types.BMD)
    md["body_type"] = b.ty
    r, v = _var4(b.r), _var4(b.v)
    systems, o = [], 0
    for c in b.counts:
        n = sum(c)
        sl = slice(o, o + n)
        playing = np.zeros(7, np.uint32)
        playing[[rg.types.STAR, rg.types.PROTOPLANET, rg.types.PLANETESIMAL, rg.types.TESTPARTICLE]] = c
        m = md[sl].copy()
        m["id"] = np.arange(1, n + 1)
        systems.append(rg.types.System(r[sl], v[sl], p[sl], m, playing))
        o += n
    cube = case["field"] == "cube"
    factor = 0.0 if cube else (5.0 if case["kind"] == "output" else 1.0)
    # at this tolerance and cadence the output interval sets the step, as in a run that
    # writes often: every try is accepted and every step is the interval
    tolerance = 1e-7 if case["integrator"] == "rk4" else 1e-10
    sim = rg.Sim(systems, integrator=case["integrator"], adaptive=case["adaptive"], tolerance=tolerance,
                 dt=CUBE_DT if cube else CADENCE, precision=case["precision"], collision_factor=factor,
                 gas=_gas() if case["gas"] else None, output_interval=0.0 if cube else CADENCE)
    n = len(b.m)
    start = SimpleNamespace(r=_pinned(n, rg.types.VAR4, r), v=_pinned(n, rg.types.VAR4, v), p=None, md=None)
    out = SimpleNamespace(r=_pinned(n, rg.types.VAR4), v=_pinned(n, rg.types.VAR4),
                          p=_pinned(n, rg.types.PARAM), md=np.zeros(n, rg.types.BMD))
    return sim, start, out


def _network(case, seed):
    """Weights in the middle of a training run: He-scaled parameters, Adam's running moments, one batch."""
    g = torch.Generator().manual_seed(int(seed))
    scale = torch.cat([torch.full((64 * 12,), math.sqrt(2.0 / 12)), torch.full((64,), 0.1),
                       torch.full((64 * 64,), math.sqrt(2.0 / 64)), torch.full((64,), 0.1),
                       torch.full((64,), math.sqrt(1.0 / 64)), torch.full((1,), 0.1)])
    master = torch.randn(scale.numel(), generator=g) * scale
    s = SimpleNamespace(master=master, w=master.bfloat16(), m=0.01 * torch.randn(scale.numel(), generator=g),
                        v=1e-4 * (0.5 + torch.rand(scale.numel(), generator=g)),
                        x=torch.randn(case["rows"], 12, generator=g))
    s.t = torch.tanh(s.x[:, 0]) + 0.3 * s.x[:, 1] * s.x[:, 2] + 0.1 * torch.randn(case["rows"], generator=g)
    return s


def prepare(case, seed):
    if case["kind"] == "train":
        s = _network(case, seed)
        for k, x in list(vars(s).items()):
            setattr(s, k, x.cuda())
        s.grad, s.loss = torch.zeros_like(s.master), torch.zeros(1, device="cuda")
        s.rows, s.kind = case["rows"], "train"
        return s
    b = _bodies(case, seed)
    if case["kind"] == "accel":
        n = len(b.m)
        dev = SimpleNamespace(kind="accel", r=torch.from_numpy(b.r).cuda(), v=torch.from_numpy(b.v).cuda(),
                              m=torch.from_numpy(b.m).cuda(), R=torch.from_numpy(b.R).cuda(),
                              id=torch.arange(1, n + 1, dtype=torch.int32, device="cuda"),
                              a=torch.zeros(n, 3, dtype=torch.float64, device="cuda"))
        g = rg.lib.AccelArgs()
        c = b.counts[0]
        for k, q in zip((rg.types.STAR, rg.types.PROTOPLANET, rg.types.PLANETESIMAL, rg.types.TESTPARTICLE), c):
            g.playing[k] = q
        g.r, g.v, g.mass, g.radius, g.id = (x.data_ptr() for x in (dev.r, dev.v, dev.m, dev.R, dev.id))
        g.accel = dev.a.data_ptr()
        g.precision = rg.lib.PRECISION[case["precision"]]
        dev.args = g
        return dev
    sim, start, out = _sim(case, b)
    return SimpleNamespace(kind=case["kind"], tries=case["tries"], sim=sim, start=start, out=out)


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _flat(a):
    return a.view(np.float64).reshape(-1, 4)


def run(s):
    if s.kind == "train":
        stream = torch.cuda.current_stream().cuda_stream
        rg.lib.mlp_grad(s.w.data_ptr(), s.x.data_ptr(), s.t.data_ptr(), s.rows, s.grad.data_ptr(), s.loss.data_ptr(),
                        stream)
        rg.lib.mlp_adam(s.master.data_ptr(), s.w.data_ptr(), s.m.data_ptr(), s.v.data_ptr(), s.grad.data_ptr(), 1000,
                        2e-3, stream=stream)
        return {"grad": s.grad, "loss": s.loss, "master": s.master, "w": s.w, "m": s.m, "v": s.v}
    if s.kind == "accel":
        s.args.stream = torch.cuda.current_stream().cuda_stream
        rg.lib.calc_accel_noalloc(s.args)
        return {"a": s.a}
    if s.kind == "output":
        I = s.sim.calc_integral(0)
        E = s.sim.energy_interacting(0)
        ev = s.sim.check_for_collision()
        s.sim.get_state(0, s.out)
        return {"integral": I, "interacting": E, "i": ev["idx1"].astype(np.int64), "j": ev["idx2"].astype(np.int64),
                "d": ev["d"].copy(), "r": _flat(s.out.r), "v": _flat(s.out.v), "p": _flat(s.out.p),
                "id": s.out.md["id"].astype(np.int64)}
    s.sim.set_states(s.start, parts="rv")
    if s.kind == "step":
        dt = s.sim.step()
        s.sim.get_states(s.out, parts="rv")
        return {"dt": dt, "r": _flat(s.out.r), "v": _flat(s.out.v)}
    s.sim.launch_tries(s.tries)
    _, halted = s.sim.synchronize()
    s.sim.get_states(s.out, parts="rv")
    return {"halted": halted, "r": _flat(s.out.r), "v": _flat(s.out.v)}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
_EVALS = {"rkf78": (11, 13), "rk4": (4, 5), "rk2": (2, 2), "euler": (1, 1)}


def _counts(case):
    """(bodies, directed interactions per evaluation) of a case; an ensemble's at its mean size."""
    def pairs(si, nsi, ni):
        return (si * (si + nsi - 1) if si else 0) + nsi * si + ni * (si + nsi)

    if case["field"] == "cube":
        return case["n_pl"], pairs(case["n_pl"], 0, 0)
    if "n_max" in case:
        n = (case["n_min"] + case["n_max"]) / 2
        return case["systems"] * n, case["systems"] * pairs(6, n - 6, 0)
    n = 1 + case["n_pp"] + case["n_pl"] + case["n_tp"]
    if case["field"] == "allpairs":
        return case["systems"] * n, case["systems"] * pairs(n - case["n_tp"], 0, case["n_tp"])
    return case["systems"] * n, case["systems"] * pairs(1 + case["n_pp"], case["n_pl"], case["n_tp"])


def work(case):
    if case["kind"] == "train":
        n = case["rows"]
        return {"bytes": 52 * n + 5057 * 30, "flops": 6 * n * (12 * 64 + 64 * 64 + 64)}
    n, pairs = _counts(case)
    if case["kind"] == "accel":
        return {"bytes": n * (24 + 8 + 8 + 4 + 24), "flops": 20 * pairs}
    if case["kind"] == "output":
        return {"bytes": n * (48 + 32 + 8) + n * (96 + 24), "flops": 10 * n * n + 10 * pairs}
    evals = _EVALS[case["integrator"]][1 if case["adaptive"] else 0] * case["tries"]
    # the state in and out of the pass, the parameters; the gravity of every evaluation
    return {"bytes": n * (128 + 32), "flops": 20 * pairs * evals}


# ---------------------------------------------------------------------------
# 64-bit results with torch alone
# ---------------------------------------------------------------------------
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _pull(sink, src, m):
    """Acceleration of the sinks (S, a, 3) by the sources (S, b, 3) of mass m (S, b); coincident pairs give nothing."""
    S, a, b = sink.shape[0], sink.shape[1], src.shape[1]
    step = max(1, int(1.0e8) // max(1, S * b))
    out = torch.zeros_like(sink)
    for k in range(0, a, step):
        d = [src[:, None, :, c] - sink[:, k:k + step, None, c] for c in range(3)]
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
        w = m[:, None, :] / (r2 * r2.sqrt())
        w = torch.where(r2 > 0, w, torch.zeros_like(w))
        for c in range(3):
            out[:, k:k + step, c] = (w * d[c]).sum(2)
    return out


def _drag(r, v, m, R, cd):
    """The acceleration f (v_gas - v) of the analytic gas disk with red's drag law."""
    g = _gas()
    eta, rho, sch = ([float(x) for x in g[k]] for k in ("eta", "rho", "sch"))
    s2 = r[..., 0] ** 2 + r[..., 1] ** 2
    s = s2.sqrt()
    speed = (1.0 / s).sqrt() * (1.0 - 2.0 * eta[0] * s ** eta[1]).sqrt()
    u = torch.stack([-r[..., 1] / s * speed - v[..., 0], r[..., 0] / s * speed - v[..., 1], -v[..., 2]], dim=-1)
    z = r[..., 2] / (sch[0] * s ** sch[1])
    dens = rho[0] * s ** rho[1] * torch.exp(-z * z)
    f = 3.0 * cd * dens * u.norm(dim=-1) / (8.0 * R * RHO)
    return f[..., None] * u


# rows of Fehlberg's 7(8) pair up to the seventh-order solution: {stage: coefficient}
_RKF = [{}, {0: 2 / 27}, {0: 1 / 36, 1: 1 / 12}, {0: 1 / 24, 2: 1 / 8}, {0: 5 / 12, 2: -25 / 16, 3: 25 / 16},
        {0: 1 / 20, 3: 1 / 4, 4: 1 / 5}, {0: -25 / 108, 3: 125 / 108, 4: -65 / 27, 5: 125 / 54},
        {0: 31 / 300, 4: 61 / 225, 5: -2 / 9, 6: 13 / 900},
        {0: 2, 3: -53 / 6, 4: 704 / 45, 5: -107 / 9, 6: 67 / 90, 7: 3},
        {0: -91 / 108, 3: 23 / 108, 4: -976 / 135, 5: 311 / 54, 6: -19 / 60, 7: 17 / 6, 8: -1 / 12},
        {0: 2383 / 4100, 3: -341 / 164, 4: 4496 / 1025, 5: -301 / 82, 6: 2133 / 4100, 7: 45 / 82, 8: 45 / 164,
         9: 18 / 41}]
_TABLEAU = {
    "rkf78": (_RKF, {0: 41 / 840, 5: 34 / 105, 6: 9 / 35, 7: 9 / 35, 8: 9 / 280, 9: 9 / 280, 10: 41 / 840}),
    "rk4": ([{}, {0: 0.5}, {1: 0.5}, {2: 1.0}], {0: 1 / 6, 1: 1 / 3, 2: 1 / 3, 3: 1 / 6}),
    "rk2": ([{}, {0: 0.5}], {1: 1.0}),
    "euler": ([{}], {0: 1.0}),
}


def exact(case, seed):
    if case["kind"] == "train":
        return _exact_train(case, seed)
    b = _bodies(case, seed)
    dev = _device()
    # systems side by side: the bodies that everything feels (stars, protoplanets) first,
    # then the planetesimals, then the test particles, each padded with massless bodies
    big = max(c[0] + c[1] for c in b.counts)
    mid = max(c[2] for c in b.counts)
    tps = max(c[3] for c in b.counts)
    where, o = [], 0
    for k, c in enumerate(b.counts):
        base = k * (big + mid + tps)
        nb, n = c[0] + c[1], sum(c)
        q = np.arange(n)
        where.append(base + np.where(q < nb, q, np.where(q < nb + c[2], big + q - nb, big + mid + q - nb - c[2])))
        o += n
    where = torch.from_numpy(np.concatenate(where))
    S, width = len(b.counts), big + mid + tps

    def spread(a, fill):
        full = torch.full((S * width,) + a.shape[1:], fill, dtype=torch.float64)
        full[where] = torch.from_numpy(a)
        return full.reshape((S, width) + a.shape[1:]).to(dev)

    r, v = spread(b.r, 1.0), spread(b.v, 0.0)
    m, R, cd = spread(b.m, 0.0), spread(b.R, 1.0), spread(b.cd, 0.0)

    def accel(r, v):
        a = torch.empty_like(r)
        a[:, :big] = _pull(r[:, :big], r[:, :big + mid], m[:, :big + mid])
        a[:, big:big + mid] = _pull(r[:, big:big + mid], r[:, :big], m[:, :big])
        if tps:
            a[:, big + mid:] = _pull(r[:, big + mid:], r[:, :big + mid], m[:, :big + mid])
        if case["gas"]:
            a[:, big:big + mid] += _drag(r[:, big:big + mid], v[:, big:big + mid], m[:, big:big + mid],
                                         R[:, big:big + mid], cd[:, big:big + mid])
        return a

    def back(a):
        return a.reshape(S * width, -1).cpu()[where].numpy()

    if case["kind"] == "accel":
        return {"a": back(accel(r, v))}
    if case["kind"] == "output":
        return _exact_output(case, r[0], v[0], m[0], big)
    rows, weights = _TABLEAU[case["integrator"]]
    dt = CUBE_DT if case["field"] == "cube" else CADENCE
    for _ in range(case["tries"] if case["kind"] == "run" else 1):
        kr, kv = [], []
        for row in rows:
            rs, vs = r.clone(), v.clone()
            for q, c in row.items():
                rs += dt * c * kr[q]
                vs += dt * c * kv[q]
            kr.append(vs)
            kv.append(accel(rs, vs))
        r = r + dt * sum(c * kr[q] for q, c in weights.items())
        v = v + dt * sum(c * kv[q] for q, c in weights.items())

    def var4(a):
        return np.concatenate([back(a), np.zeros((len(where), 1))], axis=1)

    out = {"r": var4(r), "v": var4(v)}
    out.update({"dt": dt} if case["kind"] == "step" else {"halted": None})
    return out


def _exact_output(case, r, v, m, big):
    """Barycentre, angular momentum and energy over all pairs and over the interacting ones."""
    U = torch.zeros(len(m), dtype=torch.float64, device=r.device)
    Ui = torch.zeros((), dtype=torch.float64, device=r.device)
    step = max(1, int(1.0e8) // len(m))
    for k in range(0, len(m), step):
        d = (r[k:k + step, None, :] - r[None, :, :]).norm(dim=2)
        u = torch.where(d > 0, m[None, :] / d, torch.zeros_like(d)) * m[k:k + step, None]
        U[k:k + step] = u.sum(1)
        for i in range(k, min(big, k + step)):       # each pair once, from its member that everything feels
            Ui = Ui + u[i - k, i + 1:].sum()
    M, w = m.sum(), m[:, None]
    C = torch.linalg.cross(r, v, dim=1).mul(w).sum(0)
    T = (w * v * v).sum() / 2
    I = torch.cat([(w * r).sum(0) / M, (w * v).sum(0) / M, C, (T - U.sum() / 2)[None]])
    E = torch.cat([(T - Ui)[None], C])
    return {"integral": I.cpu().numpy(), "interacting": E.cpu().numpy(), "i": None, "j": None, "d": None, "r": None,
            "v": None, "p": None, "id": None}


def _exact_train(case, seed):
    s = _network(case, seed)
    dev = _device()
    p = s.w.double().to(dev).requires_grad_(True)
    W1, b1, W2, b2, w3, b3 = torch.split(p, [64 * 12, 64, 64 * 64, 64, 64, 1])
    x, t = s.x.double().to(dev), s.t.double().to(dev)
    act = torch.nn.functional.silu
    y = act(act(x @ W1.reshape(64, 12).T + b1) @ W2.reshape(64, 64).T + b2) @ w3 + b3
    loss = ((y - t) ** 2).sum() / (2 * case["rows"])
    g = torch.autograd.grad(loss, p)[0].cpu()
    m = 0.9 * s.m.double() + 0.1 * g
    v = 0.999 * s.v.double() + 0.001 * g * g
    master = s.master.double() - 2e-3 * (m / (1 - 0.9 ** 1000)) / ((v / (1 - 0.999 ** 1000)).sqrt() + 1e-8)
    return {"grad": g.numpy(), "loss": loss.detach().cpu().reshape(1).numpy(), "master": master.numpy(), "w": None,
            "m": m.numpy(), "v": v.numpy()}
