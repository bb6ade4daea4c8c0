"""The work a program asks of this framework, as cases that can be timed and checked.

Every case goes through the public entry points of the Python front-end:
`Simulation` (the block executor), `integrate_timeblock` and `partition` (the
kernel layer, for programs that own their device memory), `Ensemble` (many
systems at once) and `learned.Trainer` (the learned Kepler starter).  Sizes are
those of the repository's synthetic workloads (glisser_gb300/synth.py), its
tests and its benchmark; the particle swarms are drawn with the same
distributions, here with torch on the GPU so that preparing a case is quick.
"""
import math

import numpy as np
import torch

import glisser_gb300 as G
from glisser_gb300 import learned as L

DEG = math.pi / 180.0
GM_DAY = 2.959122e-4            # G * Msun, au^3 / day^2
GM_YEAR = 4 * math.pi ** 2      # G * Msun, au^3 / yr^2
GIANT_M = (9.55e-4, 2.86e-4, 4.37e-5, 5.15e-5)
GIANT_A = (5.2, 9.55, 19.2, 30.1)
NEPTUNE_M = 5.15e-5

# a, e and inclination ranges of the swarms, their time step, outer limit and
# central mass.  giants, belt: the ordinary case, every particle far outside
# the planets; scattered: long eccentric orbits with pericentres among the
# planets; close: a few steps per orbit; crossers: particles on planet-crossing
# orbits, with encounter radii of three Hill radii.
SWARMS = {
    "giants": dict(planets="giants", a=(53.0, 57.0), e=(0.0, 0.3), i=10.0, dt=180.0, outer=300.0, gm=GM_DAY),
    "belt": dict(planets="neptune", a=(40.0, 50.0), e=(0.0, 0.1), i=5.0, dt=180.0, outer=300.0, gm=GM_DAY),
    "scattered": dict(planets="neptune", a=(30.0, 1000.0), e=(0.0, 0.95), i=40.0, dt=180.0, outer=1e5, gm=GM_DAY,
                      log_a=True),
    "close": dict(planets="neptune", a=(2.5, 6.0), e=(0.1, 0.6), i=20.0, dt=180.0, outer=1e5, gm=GM_DAY),
    "crossers": dict(planets="neptune", a=(20.0, 40.0), e=(0.0, 0.3), i=10.0, dt=0.2, outer=300.0, gm=GM_YEAR,
                     hill=3.0),
}
CULL = 0.5


def listed():
    return [
        # the smallest run in use (the reference's CPU-sized configuration):
        # one short block of two thousand particles, its state read back
        dict(name="belt-2k", kind="sim", swarm="belt", n=2000, steps=128),
        # the reference's own example size, 200,000 particles and four giant planets
        dict(name="giants-200k", kind="sim", swarm="giants", n=200_000, steps=512),
        # the large single-system run, a million particles
        dict(name="giants-1m", kind="sim", swarm="giants", n=1_000_000, steps=1024),
        # the reference's FP64 kick, which a user picks to compare with it
        dict(name="giants-fp64-kick", kind="block", swarm="giants", n=50_021, steps=256, kick="fp64",
             starter="series"),
        # scattered disk: steps from tiny to a sizeable part of the orbit in one warp
        dict(name="scattered-300k", kind="block", swarm="scattered", n=300_007, steps=256, kick="ff",
             starter="series"),
        # few steps per orbit, analytic starter
        dict(name="close-100k", kind="block", swarm="close", n=100_000, steps=256, kick="ff", starter="series"),
        # the same with the trained network
        dict(name="close-learned-100k", kind="block", swarm="close", n=100_000, steps=256, kick="ff",
             starter="learned"),
        # planet crossers: encounter flags, then the partition that follows each block
        dict(name="crossers-2m", kind="block", swarm="crossers", n=2_000_000, steps=100, kick="ff",
             starter="series"),
        # the ensembles workload at a quarter of its particles, state read back each block
        dict(name="ensembles-256", kind="ensemble", systems=256, particles=1_500_000, steps=512),
        # a handful of small systems, ragged counts
        dict(name="ensembles-16", kind="ensemble", systems=16, particles=9_000, steps=256),
        # the partition alone, as a program with its own buffers calls it after each block
        dict(name="partition-1m", kind="partition", n=1_000_003, flagged=0.05),
        # Adam steps of the learned starter's network
        dict(name="learned-train", kind="train", samples=200_000, batch=16384, steps=100),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("sim", "sim", "block", "block", "block", "ensemble", "ensemble", "partition", "train"))
    if kind == "sim":
        return dict(kind=kind, swarm=rng.choice(("belt", "giants")), n=_log_int(rng, 500, 800_000),
                    steps=rng.randrange(65, 769))
    if kind == "block":
        swarm = rng.choice(("giants", "scattered", "close", "crossers"))
        return dict(kind=kind, swarm=swarm, n=_log_int(rng, 1000, 150_000 if swarm == "close" else 600_000),
                    steps=rng.randrange(33, 321), kick=rng.choice(("ff", "ff", "fp64")),
                    starter=rng.choice(("series", "learned")) if swarm == "close" else "series")
    if kind == "ensemble":
        systems = _log_int(rng, 4, 256)
        return dict(kind=kind, systems=systems, particles=systems * _log_int(rng, 200, 5000),
                    steps=rng.randrange(65, 513))
    if kind == "partition":
        return dict(kind=kind, n=_log_int(rng, 5000, 4_000_000), flagged=round(rng.uniform(0.0, 0.5), 3))
    return dict(kind=kind, samples=200_000, batch=128 * _log_int(rng, 16, 512), steps=rng.randrange(20, 200))


# ---------------------------------------------------------------------------
# Inputs


def _device():
    return torch.device("cuda:0")


def _to_cartesian(mu, el):
    """Elements (a, e, i, node, peri, M), each [n] -> r, v [3, n]."""
    a, e, inc, node, peri, M = el
    E = M + 0.85 * e * torch.sign(torch.sin(M))
    for _ in range(12):
        f = E - e * torch.sin(E) - M
        fp = 1 - e * torch.cos(E)
        d = -f / fp
        d = -f / (fp + 0.5 * d * e * torch.sin(E))
        E = E + d
    q = torch.sqrt(1 - e * e)
    s, c = torch.sin(E), torch.cos(E)
    n = torch.sqrt(mu / a ** 3)
    x, y = a * (c - e), a * q * s
    ed = n / (1 - e * c)
    vx, vy = -a * s * ed, a * q * c * ed
    so, co, sn, cn, si, ci = (torch.sin(peri), torch.cos(peri), torch.sin(node), torch.cos(node), torch.sin(inc),
                              torch.cos(inc))
    p = torch.stack([cn * co - sn * so * ci, sn * co + cn * so * ci, so * si])
    w = torch.stack([-cn * so - sn * co * ci, -sn * so + cn * co * ci, co * si])
    return p * x + w * y, p * vx + w * vy


def _swarm(sw, n, gen):
    """n particles of a swarm: r, v [3, n] on the GPU."""
    u = torch.rand((6, n), dtype=torch.float64, device=_device(), generator=gen)
    lo, hi = sw["a"]
    a = torch.exp(math.log(lo) + u[0] * math.log(hi / lo)) if sw.get("log_a") else lo + u[0] * (hi - lo)
    e = sw["e"][0] + u[1] * (sw["e"][1] - sw["e"][0])
    ang = 2 * math.pi
    return _to_cartesian(sw["gm"], (a, e, u[2] * sw["i"] * DEG, u[3] * ang, u[4] * ang, u[5] * ang))


def _planets(kind, gm, rng, scatter=False):
    """m [npl] with the Sun first, elements [npl - 1, 6]."""
    if kind == "neptune":
        return np.array([gm, NEPTUNE_M * gm]), np.array([[30.0, 0, 0, 0, 0, rng.uniform(0, 2 * math.pi)]])
    ms = np.array(GIANT_M) * (rng.uniform(0.9, 1.1, 4) if scatter else 1.0)
    a = np.array(GIANT_A) * (rng.uniform(0.95, 1.05, 4) if scatter else 1.0)
    el = np.stack([a, rng.uniform(0, 0.05, 4), rng.uniform(0, 2 * DEG, 4), *rng.uniform(0, 2 * math.pi, (3, 4))], 1)
    return np.concatenate([[gm], ms * gm]), el


def _planet_state(m, el):
    """Heliocentric r, v [npl, 3] of the planets, the Sun at the origin."""
    r, v = [np.zeros(3)], [np.zeros(3)]
    for j, row in enumerate(el):
        x, w = _to_cartesian(m[0] + m[j + 1], [torch.tensor([c], dtype=torch.float64) for c in row])
        r.append(x[:, 0].numpy())
        v.append(w[:, 0].numpy())
    return np.array(r), np.array(v)


def _planet_log(m, el, dt, steps):
    """Per step h0 and the planets' positions on their Kepler orbits,
    [steps + 1, npl, 3] (record 0 is the start)."""
    t = torch.arange(steps + 1, dtype=torch.float64) * dt
    log = np.zeros((steps + 1, len(m), 3))
    for j, row in enumerate(el):
        mu = m[0] + m[j + 1]
        one = torch.ones_like(t)
        M = row[5] + math.sqrt(mu / row[0] ** 3) * t
        r, _ = _to_cartesian(mu, [one * c for c in row[:5]] + [M])
        r = r.numpy().T
        log[:, j + 1] = r
        log[:, 0] -= m[j + 1] * r / np.linalg.norm(r, axis=1, keepdims=True) ** 3
    return log


def _radii(m, el, hill):
    rh = np.full(len(m), CULL)
    if hill:
        rh[1:] = hill * el[:, 0] * (1 - el[:, 1]) * (m[1:] / (3 * m[0])) ** (1.0 / 3)
    return rh


def _config(steps, dt, outer):
    return ("Time-Step %r\nTime-Block-Size %d\nFinal-Time 1e12\nOuter-Limit %r\nCull-Radius %r\n"
            "Input-File unused\nOutput-Folder unused\n" % (dt, steps, outer, CULL))


def _host(x):
    """[3, n] on the GPU -> [n, 3] on the host."""
    return np.ascontiguousarray(x.t().contiguous().cpu().numpy())


class _Particles:
    """A program's own particle buffers: the arrays of glisser_particles."""

    def __init__(self, n):
        dev = _device()
        self.f = torch.zeros((9, n), dtype=torch.float64, device=dev)
        self.flags = torch.zeros(n, dtype=torch.int16, device=dev)
        self.dti = torch.zeros(n, dtype=torch.int32, device=dev)
        self.id = torch.arange(n, dtype=torch.int32, device=dev)
        self.view = G.ParticlesDev(*[self.f[k].data_ptr() for k in range(9)], self.flags.data_ptr(),
                                   self.dti.data_ptr(), self.id.data_ptr())

    def out(self):
        return dict(state=self.f, flags=self.flags, deathtime_index=self.dti, id=self.id)


def _samples(n, seed):
    """Kepler solves of close-orbit drifts: the network's features and target."""
    gen = torch.Generator(device=_device()).manual_seed(seed + 77)
    sw = SWARMS["close"]
    r, v = _swarm(sw, n, gen)
    mu, dt = sw["gm"], sw["dt"]
    r0 = r.norm(dim=0)
    u = (r * v).sum(0)
    alpha = 2 * mu / r0 - (v * v).sum(0)
    s, _ = _solve(r0, u, alpha, mu, dt, True)
    tau = dt * torch.sqrt(mu / r0 ** 3)
    feat = torch.stack([torch.log(tau), u / torch.sqrt(mu * r0), alpha * r0 / mu], 1)
    return feat.float().cpu().numpy(), (torch.log(s * r0 / dt) / tau).float().cpu().numpy()


def _trainer(samples, seed):
    tr = L.Trainer(samples, seed=7)
    feat, target = _samples(samples, seed)
    tr.add_samples(feat, target)
    tr.fit_norm()
    return tr


def _ensemble_inputs(case, seed):
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device=_device()).manual_seed(seed)
    # the systems' sizes belong to the case, their orbits to the seed
    w = np.exp(np.random.default_rng(case["systems"]).normal(0.0, 0.6, case["systems"]))
    counts = np.maximum(1, np.round(w / w.sum() * case["particles"])).astype(int)
    r, v = _swarm(SWARMS["belt"], int(counts.sum()), gen)
    planets = [_planets("giants", GM_DAY, rng, True) for _ in counts]
    return counts, [p[0] for p in planets], [_planet_state(*p) for p in planets], r, v


def _sim_inputs(case, seed):
    sw = SWARMS[case["swarm"]]
    m, el = _planets(sw["planets"], sw["gm"], np.random.default_rng(seed))
    pr, pv = _planet_state(m, el)
    r, v = _swarm(sw, case["n"], torch.Generator(device=_device()).manual_seed(seed))
    return sw, m, pr, pv, r, v


def _block_inputs(case, seed):
    sw = SWARMS[case["swarm"]]
    m, el = _planets(sw["planets"], sw["gm"], np.random.default_rng(seed))
    log = _planet_log(m, el, sw["dt"], case["steps"])
    r, v = _swarm(sw, case["n"], torch.Generator(device=_device()).manual_seed(seed))
    a = _acceleration(r, torch.tensor(log[0], device=_device()), m)
    return sw, m, log, _radii(m, el, sw.get("hill")), r, v, a


def _partition_inputs(case, seed):
    n = case["n"]
    gen = torch.Generator(device=_device()).manual_seed(seed)
    p = _Particles(n)
    p.f.normal_(generator=gen)
    u = torch.rand(n, device=_device(), generator=gen)
    # of the flagged particles half are in an encounter (planet id in the high
    # byte) and half left the run
    flags = torch.where(u < case["flagged"] / 2, 0x0401, torch.where(u < case["flagged"], 0x0080, 0))
    p.flags.copy_(flags.to(torch.int16))
    p.dti.copy_(torch.randint(0, 2048, (n,), device=_device(), generator=gen).to(torch.int32))
    return p


def prepare(case, seed):
    kind = case["kind"]
    st = dict(kind=kind)
    if kind == "sim":
        sw, m, pr, pv, r, v = _sim_inputs(case, seed)
        sim = G.Simulation(_config(case["steps"], sw["dt"], sw["outer"]))
        sim.set_planets(m, pr, pv)
        sim.set_particles(_host(r), _host(v))
        sim.init()
        st.update(sim=sim)
    elif kind == "block":
        sw, m, log, rh, r, v, a = _block_inputs(case, seed)
        n, dev = case["n"], _device()
        p = _Particles(n)
        rec = torch.zeros(((case["steps"] + 1) // 2 * 2, len(m), 3), dtype=torch.float64)
        rec[:case["steps"]] = torch.tensor(log[1:])
        keep = dict(log=rec.to(dev), m=torch.tensor(m, device=dev), rh=torch.tensor(rh, device=dev),
                    pid=torch.arange(len(m), dtype=torch.int32, device=dev),
                    index=torch.zeros(n, dtype=torch.int32, device=dev),
                    hid=torch.zeros(n, dtype=torch.int32, device=dev),
                    hfl=torch.zeros(n, dtype=torch.int16, device=dev),
                    hdti=torch.zeros(n, dtype=torch.int32, device=dev),
                    ctr=torch.zeros(4, dtype=torch.int32, device=dev))
        blk = G.PlanetBlockDev(keep["log"].data_ptr(), keep["m"].data_ptr(), keep["pid"].data_ptr(),
                               keep["rh"].data_ptr(), len(m), case["steps"], rec.shape[0], 0)
        c = keep["ctr"].data_ptr()
        ho = G.HandoffDev(c, keep["index"].data_ptr(), keep["hid"].data_ptr(), keep["hfl"].data_ptr(),
                          keep["hdti"].data_ptr(), n, 0, c + 4, None, None, None, None)
        mlp = 0
        if case["starter"] == "learned":
            tr = _trainer(100_000, 5)
            tr.train(2000, batch=16384, lr=1e-2, seed=3)
            mlp = tr.device_weights()
            keep["trainer"] = tr
        sp = G.StepParams(sw["dt"], sw["outer"], G.STARTER_LEARNED if mlp else G.STARTER_SERIES,
                          G.ENCOUNTERS_KILL, mlp, 0.0, G.KICK_FP64 if case["kick"] == "fp64" else
                          G.KICK_FLOAT_FLOAT)
        st.update(p=p, start=torch.cat([r, v, a]), keep=keep, blk=blk, ho=ho, sp=sp, n=n)
        if sw.get("hill"):
            st.update(q=_Particles(n), scratch=torch.zeros(G.partition_scratch_bytes(n), dtype=torch.uint8,
                                                           device=dev))
    elif kind == "ensemble":
        counts, ms, pl, r, v = _ensemble_inputs(case, seed)
        r, v = _host(r), _host(v)
        ens = G.Ensemble(_config(case["steps"], 180.0, 300.0), len(counts))
        at = 0
        for s, k in enumerate(counts):
            ens.set_system(s, ms[s], pl[s][0], pl[s][1], r[at:at + k], v[at:at + k])
            at += k
        ens.init()
        st.update(ens=ens, r=np.zeros((at, 3)), v=np.zeros((at, 3)), flags=np.zeros(at, np.uint16))
    elif kind == "partition":
        p, n = _partition_inputs(case, seed), case["n"]
        st.update(p=p, q=_Particles(n), n=n, ctr=torch.zeros(2, dtype=torch.int32, device=_device()),
                  scratch=torch.zeros(G.partition_scratch_bytes(n), dtype=torch.uint8, device=_device()))
    else:
        st.update(tr=_trainer(case["samples"], seed), batch=case["batch"], steps=case["steps"])
    return st


def run(st):
    kind = st["kind"]
    if kind == "sim":
        st["sim"].loop()
        return st["sim"].particles()
    if kind == "block":
        # a block from the program's checkpoint buffer
        p = st["p"]
        p.f.copy_(st["start"])
        p.flags.zero_()
        st["keep"]["ctr"].zero_()
        G.integrate_timeblock(p.view, st["n"], st["blk"], st["sp"], st["ho"])
        if "q" not in st:
            return p.out()
        c = st["keep"]["ctr"]
        G.partition(p.view, st["q"].view, st["n"], st["scratch"].data_ptr(), c.data_ptr() + 8, c.data_ptr() + 12)
        return dict(st["q"].out(), counts=c)
    if kind == "ensemble":
        st["ens"].step()
        r, v, flags = st["ens"].get_state(st["r"], st["v"], st["flags"])
        return dict(r=r, v=v, flags=flags)
    if kind == "partition":
        c = st["ctr"]
        G.partition(st["p"].view, st["q"].view, st["n"], st["scratch"].data_ptr(), c.data_ptr(), c.data_ptr() + 4)
        return dict(st["q"].out(), counts=c)
    losses = st["tr"].train(st["steps"], batch=st["batch"], lr=3e-3, seed=1)
    return dict(losses=losses, params=st["tr"].params)


def work(case):
    """State in and out once (90 bytes a particle each way); per particle-step
    the operations of one universal-variable drift with a single Newton
    evaluation and 18 for each planet's pull."""
    kind = case["kind"]
    if kind == "partition":
        return dict(bytes=2 * 90.0 * case["n"], flops=0.0)
    if kind == "train":
        # forward and backward products of the 3-32-32-1 network
        per = 2 * 3 * (3 * 32 + 32 * 32 + 32)
        return dict(bytes=16.0 * case["batch"] * case["steps"], flops=float(per) * case["batch"] * case["steps"])
    n = case["particles"] if kind == "ensemble" else case["n"]
    giants = kind == "ensemble" or SWARMS[case["swarm"]]["planets"] == "giants"
    return dict(bytes=2 * 90.0 * n, flops=(113.0 + 18 * (4 if giants else 1)) * n * case["steps"])


# ---------------------------------------------------------------------------
# The same results in plain 64-bit arithmetic


def _stumpff(x, terms):
    c2, c3 = torch.zeros_like(x), torch.zeros_like(x)
    for k in range(terms - 1, -1, -1):
        c2 = 1.0 / math.factorial(2 * k + 2) - x * c2
        c3 = 1.0 / math.factorial(2 * k + 3) - x * c3
    return c2, c3


def _solve(r0, u, alpha, mu, dt, wide):
    """The universal anomaly s of a drift by dt, and its G-functions."""
    T = dt / r0
    k = mu - alpha * r0
    terms = 20 if wide else 6

    def g_of(s):
        c2, c3 = _stumpff(alpha * s * s, terms)
        g2, g3 = s * s * c2, s * s * s * c3
        return 1 - alpha * g2, s - alpha * g3, g2, g3

    if wide:
        s = T / (1 + 0.5 * T * u / r0).clamp(min=0.5)
        for _ in range(9):      # Laguerre
            g0, g1, g2, g3 = g_of(s)
            f = r0 * g1 + u * g2 + mu * g3 - dt
            fp = r0 * g0 + u * g1 + mu * g2
            fpp = k * g1 + u * g0
            disc = torch.sqrt((16 * fp * fp - 20 * f * fpp).abs())
            s = s - 5 * f / (fp + disc)
    else:
        X = 0.5 * u * T / r0
        s = T * (1 - X)
    for _ in range(2 if wide else 3):
        g0, g1, g2, g3 = g_of(s)
        f = r0 * g1 + u * g2 + (mu * g3 - dt)
        s = s - f / (r0 * g0 + u * g1 + mu * g2)
    return s, g_of(s)


def _drift(r, v, mu, dt, wide):
    r0 = r.norm(dim=0)
    u = (r * v).sum(0)
    alpha = 2 * mu / r0 - (v * v).sum(0)
    _, (g0, g1, g2, g3) = _solve(r0, u, alpha, mu, dt, wide)
    nr = r + (v * (dt - mu * g3) - r * (mu / r0 * g2))
    n0 = nr.norm(dim=0)
    return nr, v - (r * (mu * g1 / (r0 * n0)) + v * (mu * g2 / n0))


def _acceleration(r, rec, m):
    """rec: h0 and planet positions, [npl, 3] or (per particle) [npl, 3, n]."""
    shared = rec.dim() == 2
    a = (rec[0][:, None] if shared else rec[0]).expand_as(r).clone()
    for j in range(1, rec.shape[0]):
        d = r - (rec[j][:, None] if shared else rec[j])
        a -= d * (m[j] / (d * d).sum(0) ** 1.5)
    return a


def _wh_block(r, v, a, record, steps, m, mu, rh2, outer2, dt, wide):
    """Kick-drift-kick over a block; a particle inside a radius stops there."""
    live = torch.ones(r.shape[1], dtype=torch.bool, device=r.device)
    for s in range(steps):
        rec = record(s)
        w = v + a * (0.5 * dt)
        nr, w = _drift(r, w, mu, dt, wide)
        na = _acceleration(nr, rec, m)
        w = w + na * (0.5 * dt)
        out = (nr * nr).sum(0)
        hit = (out < rh2[0]) | (out > outer2)
        for j in range(1, rec.shape[0]):
            d = nr - (rec[j][:, None] if rec.dim() == 2 else rec[j])
            hit |= (d * d).sum(0) < rh2[j]
        r, v, a = torch.where(live, nr, r), torch.where(live, w, v), torch.where(live, na, a)
        live = live & ~hit
    return r, v, a, live


def _planet_wh(m, r, v, dt, steps):
    """The planets' own Wisdom-Holman map in Jacobi coordinates for many
    systems at once: m [S, npl], r, v [S, npl, 3] -> h0 and positions per step
    [steps, S, npl, 3], and the start's h0 [S, 3]."""
    m, r, v = m.copy(), r.copy(), v.copy()
    npl = m.shape[1]
    eta = np.cumsum(m, 1)

    def jacobi(x):
        y = x.copy()
        y[:, 0] = 0
        acc = np.zeros_like(x[:, 0])
        for i in range(2, npl):
            acc = acc + x[:, i - 1] * m[:, i - 1, None]
            y[:, i] = x[:, i] - acc / eta[:, i - 1, None]
        return y

    def helio(y):
        x = y.copy()
        acc = np.zeros_like(y[:, 0])
        for i in range(2, npl):
            acc = acc + y[:, i - 1] * (m[:, i - 1] / eta[:, i - 1])[:, None]
            x[:, i] = y[:, i] + acc
        return x

    def cube(x):
        return ((x * x).sum(-1) ** -1.5)[..., None]

    def accelerations(x, y):
        ir, ij = cube(x[:, 1:]), cube(y[:, 1:])
        pull = x[:, 1:] * m[:, 1:, None] * ir
        h0 = -pull.sum(1)
        acc = np.zeros_like(x)
        acc[:, 1:] = -pull[:, 1:].sum(1, keepdims=True)
        accum = np.zeros_like(x[:, 0])
        for i in range(2, npl):
            acc[:, i] += (y[:, i] * ij[:, i - 1] - x[:, i] * ir[:, i - 1]) * m[:, :1]
            accum = accum + y[:, i] * ij[:, i - 1] * (m[:, i] * m[:, 0] / eta[:, i - 1])[:, None]
            acc[:, i] += accum
        for i in range(1, npl - 1):
            for j in range(i + 1, npl):
                d = x[:, j] - x[:, i]
                c = cube(d)
                acc[:, j] -= d * c * m[:, i, None]
                acc[:, i] += d * c * m[:, j, None]
        return h0, acc

    mu = np.zeros_like(m)
    mu[:, 1:] = m[:, :1] * eta[:, 1:] / eta[:, :-1]
    y = jacobi(r)
    first, acc = accelerations(r, y)
    log = np.zeros((steps,) + r.shape)
    for s in range(steps):
        v = v + acc * (0.5 * dt)
        w = jacobi(v)
        q, p = y[:, 1:], w[:, 1:]
        dist = np.sqrt((q * q).sum(-1))
        a = 1 / (2 / dist - (p * p).sum(-1) / mu[:, 1:])
        n = np.sqrt(mu[:, 1:] / a ** 3)
        ec, es = 1 - dist / a, (q * p).sum(-1) / (n * a * a)
        dm = dt * n
        de = dm - es + es * np.cos(dm) + ec * np.sin(dm)
        for _ in range(7):
            sn, cs = np.sin(de), np.cos(de)
            de = de - (de - ec * sn + es * (1 - cs) - dm) / (1 - ec * cs + es * sn)
        sn, cs = np.sin(de), np.cos(de)
        fp = 1 - ec * cs + es * sn
        y, w = y.copy(), w.copy()
        y[:, 1:] = q * (1 + a * (cs - 1) / dist)[..., None] + p * (dt + (sn - de) / n)[..., None]
        w[:, 1:] = q * (-n * sn * a / (dist * fp))[..., None] + p * (1 + (cs - 1) / fp)[..., None]
        r, v = helio(y), helio(w)
        h0, acc = accelerations(r, y)
        v = v + acc * (0.5 * dt)
        log[s] = r
        log[s, :, 0] = h0
    return log, first


def exact(case, seed):
    kind = case["kind"]
    dev = _device()
    if kind == "sim":
        sw, m, pr, pv, r, v = _sim_inputs(case, seed)
        log, h0 = _planet_wh(m[None], pr[None], pv[None], sw["dt"], case["steps"])
        log = torch.tensor(log[:, 0], device=dev)
        first = torch.tensor(pr, device=dev)
        first[0] = torch.tensor(h0[0])
        r, v, _, live = _wh_block(r, v, _acceleration(r, first, m), lambda s: log[s], case["steps"], m, m[0],
                                  np.full(len(m), CULL ** 2), sw["outer"] ** 2, sw["dt"], False)
        # a particle that left the run moves to the back of the arrays
        order = torch.argsort((~live).to(torch.int8), stable=True)
        return dict(r=_host(r[:, order]), v=_host(v[:, order]), id=None, flags=None, deathtime=None,
                    deathtime_index=None)
    if kind == "block":
        sw, m, log, rh, r, v, a = _block_inputs(case, seed)
        log = torch.tensor(log, device=dev)
        wide = case["swarm"] in ("scattered", "close")
        r, v, a, live = _wh_block(r, v, a, lambda s: log[s + 1], case["steps"], m, m[0], rh ** 2, sw["outer"] ** 2,
                                  sw["dt"], wide)
        f = torch.cat([r, v, a])
        if sw.get("hill"):
            f = f[:, torch.argsort((~live).to(torch.int8), stable=True)]
        return dict(state=f, flags=None, deathtime_index=None, id=None)
    if kind == "ensemble":
        counts, ms, pl, r, v = _ensemble_inputs(case, seed)
        m = np.array(ms)
        log, h0 = _planet_wh(m, np.array([p[0] for p in pl]), np.array([p[1] for p in pl]), 180.0, case["steps"])
        first = np.array([p[0] for p in pl])
        first[:, 0] = h0
        which = torch.repeat_interleave(torch.arange(len(counts)), torch.tensor(counts)).to(dev)

        def spread(x):          # [S, npl, 3] -> [npl, 3, n]
            return torch.as_tensor(x, device=dev).permute(1, 2, 0).contiguous()[:, :, which]

        log = torch.tensor(log, device=dev)
        mass = torch.tensor(m.T.copy(), device=dev)[:, which]
        r, v, _, _ = _wh_block(r, v, _acceleration(r, spread(first), mass), lambda s: spread(log[s]), case["steps"],
                               mass, GM_DAY, np.full(5, CULL ** 2), 300.0 ** 2, 180.0, False)
        return dict(r=_host(r), v=_host(v), flags=None)
    if kind == "partition":
        p = _partition_inputs(case, seed)
        order = torch.argsort(torch.where(p.flags == 0, 0, torch.where((p.flags & 0xFE) == 0, 1, 2)), stable=True)
        return dict(state=p.f[:, order], flags=None, deathtime_index=None, id=None, counts=None)
    # the network's weights are rounded to BF16 at every step: a run in 64-bit
    # arithmetic rounds some of them the other way and is another run
    return None
