"""The work a user of this library has it do, as cases that can be timed.

Each case is one whole pass through the public Python entry points (which make
the C calls that a Fortran host makes): a system goes in, some steps are made,
states, records or gradients come back. The library holds one resident system,
so a pass uploads its own. Systems come from the package's seeded generator,
with the element distributions of its benchmark workloads: a central mass, one
to eight planets, massless particles. Steps are 8 days unless a case says
otherwise, encounters are screened at 3 Hill radii, central impacts at
0.005 AU, adaptive integrators run at a tolerance of 1e-12.
"""
import math

import numpy as np
import torch

from mercuda_b200.adjoint import hybrid_trajectory, mvs_trajectory
from mercuda_b200.backend import EVENT_DTYPE, Backend, Batch
from mercuda_b200.system import make_system, mce_init

RCEN = 0.005
RMAX = 100.0
TOL = 1e-12
K2 = 2.959122082855911e-4
LIGHT = 299792458.0 * 86400.0 / 1.495978707e11   # AU/day


def listed():
    return [
        # a handful of particles followed step by step with every record looked
        # at as it happens: launches and latency are all there is
        dict(name="steps_200", kind="steps", particles=200, planets=4, steps=46, h=8.0, near=0.01, yar=False),
        # one year of the standard small run in one call
        dict(name="run_10k", kind="run", particles=10_000, planets=8, steps=46, h=8.0, near=0.0, yar=False),
        # ten years of the large run (1% near a planet, so records come back),
        # from and to page-locked buffers
        dict(name="run_1M", kind="run", particles=1_000_000, planets=8, steps=457, h=8.0, near=0.01, yar=False),
        # the step-by-step host loop on an odd size, with Yarkovsky forces
        dict(name="steps_300k", kind="steps", particles=300_001, planets=8, steps=46, h=8.0, near=0.01, yar=True),
        # what an output interval asks for: physical coordinates through the
        # symplectic corrector, the energy check, the ejection screen
        dict(name="output_100k", kind="output", particles=100_000, planets=8, h=8.0, near=0.0, yar=False),
        # close encounters followed through the hybrid integrator
        dict(name="hybrid_100k", kind="hybrid", particles=100_000, planets=8, steps=10, h=8.0),
        # dust and small bodies with radiation forces and relativity, and plain
        # gravity by the integrator made for it
        dict(name="radau_100k", kind="adaptive", method="RADAU", particles=100_000, planets=8, days=60.0),
        dict(name="bs_20k", kind="adaptive", method="BS", particles=20_001, planets=8, days=60.0),
        dict(name="bs2_100k", kind="adaptive", method="BS2", particles=100_000, planets=8, days=60.0),
        # many small independent systems at once, in the launch shape that a
        # program keeps from its earlier runs
        dict(name="batch_1024", kind="batch", systems=1024, nmin=10, nmax=5000, steps=457, near=0.0),
        # sensitivities of 1,000 steps to the initial states and drift rates
        dict(name="adjoint_100k", kind="adjoint", particles=100_000, planets=8, steps=1000, every=50, h=8.0),
        # the same through encounters
        dict(name="hybrid_adjoint_20k", kind="hybrid_adjoint", particles=20_000, planets=8, steps=5, every=5,
             h=8.0),
    ]


def _log(rng, lo, hi):
    """An integer, often odd, spread over the logarithm of lo .. hi."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps", "run", "run", "output", "hybrid", "adaptive", "adaptive", "batch", "adjoint"])
    planets = rng.randint(1, 8)
    h = rng.choice([8.0, 8.0, -8.0, rng.uniform(4.0, 8.0)])
    near = rng.choice([0.0, 0.01])
    if kind == "steps":
        return dict(kind=kind, particles=_log(rng, 100, 600_000), planets=planets, steps=rng.randint(16, 46), h=h,
                    near=near, yar=rng.random() < 0.4)
    if kind == "run":
        return dict(kind=kind, particles=_log(rng, 100, 1_000_000), planets=planets, steps=_log(rng, 16, 457), h=h,
                    near=near, yar=rng.random() < 0.3)
    if kind == "output":
        return dict(kind=kind, particles=_log(rng, 1_000, 600_000), planets=planets, h=h, near=near,
                    yar=rng.random() < 0.3)
    if kind == "hybrid":
        return dict(kind=kind, particles=_log(rng, 1_000, 100_000), planets=planets, steps=rng.randint(3, 10), h=8.0)
    if kind == "adaptive":
        return dict(kind=kind, method=rng.choice(["RADAU", "BS", "BS2"]), particles=_log(rng, 500, 100_000),
                    planets=planets, days=rng.choice([1, 1, -1]) * rng.uniform(20.0, 60.0))
    if kind == "batch":
        return dict(kind=kind, systems=_log(rng, 16, 1024), nmin=10, nmax=_log(rng, 100, 5000),
                    steps=_log(rng, 31, 457), near=near)
    return dict(kind=kind, particles=_log(rng, 500, 100_000), planets=planets, steps=_log(rng, 50, 1000),
                every=rng.choice([25, 50, 64]), h=h)


# ------------------------------------------------------------------- inputs
def _yar(n, seed):
    """Yarkovsky drift coefficients, log-uniform in size, of either sign."""
    rng = np.random.default_rng((seed, 7))
    return np.exp(rng.uniform(math.log(1e-15), math.log(1e-13), n)) * rng.choice([-1.0, 1.0], n)


def _barycentric(s):
    """Velocities of a hybrid run: relative to the centre of mass."""
    s.v -= (s.m[1:, None] * s.v[1:]).sum(axis=0) / s.m.sum()
    return s


def _system(case, seed):
    kind = case["kind"]
    h = case.get("h", 8.0)
    s = make_system(seed=seed, n_particles=case["particles"], nplanets=case["planets"],
                    near_fraction=case.get("near", 0.0), h=h)
    npart = s.n - s.nbig
    if kind in ("hybrid", "hybrid_adjoint"):
        s = _barycentric(mce_init(s, h, 3.0))
    if case.get("yar") or kind in ("adjoint", "hybrid_adjoint"):
        s.ngf[s.nbig:, 4] = _yar(npart, seed)
    if kind == "adaptive" and case["method"] != "BS2":   # BS2 is for forces of position alone
        s.ngf[s.nbig:, 3] = np.random.default_rng((seed, 3)).uniform(0.01, 0.3, npart)
        s.ngf[s.nbig:, 4] = _yar(npart, seed)
        s.pn = 1
    return s


def _sizes(case):
    """Particles of each system of a batch: log-uniform, the same for every seed."""
    rng = np.random.default_rng(case["systems"])
    return np.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"]), case["systems"])).astype(int)


def _batch_systems(case, seed):
    sizes = _sizes(case)
    planets = np.random.default_rng(case["nmax"]).integers(1, 9, len(sizes))
    rng = np.random.default_rng(seed)
    h = rng.uniform(4.0, 16.0, len(sizes))
    return [make_system(seed=int(rng.integers(1 << 30)), n_particles=int(n), nplanets=int(p),
                        near_fraction=case["near"], h=float(hs)) for n, p, hs in zip(sizes, planets, h)], h


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    t.numpy()[...] = a
    return t.numpy()


def _tables(case):
    """The tables a program keeps its encounter records in: room for several
    times what these systems give, unused rows zero."""
    if case["kind"] == "adaptive":
        room = case["particles"] * abs(case["days"])
    else:
        room = _particles(case) * case["steps"]
    room = 256 + int(room / 400)
    return dict(records=np.zeros(room, dtype=EVENT_DTYPE), labels=np.zeros((2, room), dtype=np.int32))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        systems, h = _batch_systems(case, seed)
        return dict(case=case, systems=systems, h=h, **_tables(case))
    s = _system(case, seed)
    state = dict(case=case, system=s, flag=s.ngflag)
    if kind in ("adjoint", "hybrid_adjoint"):
        dev, nb = torch.device("cuda"), s.nbig
        state["inputs"] = [torch.tensor(a, device=dev, requires_grad=True)
                           for a in (s.x[nb:], s.v[nb:], s.ngf[nb:, 4])]
        state["big"] = (s.m[:nb].copy(), s.x[:nb].copy(), s.v[:nb].copy())
        return state
    if kind == "run":
        for name in ("m", "x", "v", "ngf", "rce", "rphys"):
            setattr(s, name, _pinned(getattr(s, name)))
        state["out"] = (_pinned(np.zeros((s.n, 3))), _pinned(np.zeros((s.n, 3))))
    if kind != "output":
        state.update(_tables(case))
    b = Backend({"hybrid": "HYBRID", "adaptive": case.get("method")}.get(kind, "MVS"))
    b.configure()
    state["backend"] = b
    return state


# --------------------------------------------------------------------- runs
def _kept(state, events, *labels):
    """The pass's records (and what labels them: steps, systems) put into the
    program's tables; the tables' columns."""
    table, n = state["records"], len(events)
    if n > len(table):
        raise RuntimeError("more records than the tables have room for")
    table[:n] = events
    for k, values in enumerate(labels):
        state["labels"][k, :n] = values
    return dict(records=n, labels=state["labels"], **{k: table[k] for k in EVENT_DTYPE.names})


def _run_steps(state):
    """The host loop: a step, the records of the step, the next step."""
    b, s, c = state["backend"], state["system"], state["case"]
    b.upload(s, state["flag"])
    t, h, got = 0.0, c["h"], []
    for k in range(c["steps"]):
        b.step(t, h, dtflag=2 if k else 0)
        t = t + h
        got.append(b.events(t, h, RCEN))
    x, v = b.download()
    return dict(x=x, v=v, count=np.array([len(e) for e in got]), **_kept(state, np.concatenate(got)))


def _run_run(state):
    b, s, c = state["backend"], state["system"], state["case"]
    events, steps, x, v = b.mvs_run(s, 0.0, c["h"], c["steps"], RCEN, ngflag=state["flag"], out=state["out"])
    return dict(x=x, v=v, **_kept(state, events, steps))


def _run_output(state):
    b, s, c = state["backend"], state["system"], state["case"]
    b.upload(s, state["flag"])
    b.step(0.0, c["h"], dtflag=0)
    x, v = b.export(c["h"], physical=True)
    e, l2 = b.energy(c["h"], physical=True)
    return dict(x=x, v=v, energy=e, l2=l2, ejected=b.ejections(c["h"], False, RMAX))


def _run_hybrid(state):
    b, s, c = state["backend"], state["system"], state["case"]
    b.upload(s, state["flag"])
    t, h, carry, pairs, near, hits = 0.0, c["h"], {"dtflag": 0}, [], [], []
    for _ in range(c["steps"]):
        events, npair = b.hybrid_step(s, t, h, TOL, carry, RCEN)
        t = t + h
        near.append(events)
        pairs.append(npair)
        hits.append(len(b.events(t, h, RCEN)))
    x, v = b.download()
    return dict(x=x, v=v, pairs=np.array(pairs), hits=np.array(hits), **_kept(state, np.concatenate(near)))


def _run_adaptive(state):
    b, s, c = state["backend"], state["system"], state["case"]
    b.upload(s, state["flag"])
    events, where, h, steps = b.hvar_run(0.0, c["days"], math.copysign(2.0, c["days"]), TOL, RCEN)
    x, v = b.download()
    return dict(x=x, v=v, h=h, steps=steps, **_kept(state, events, where))


def _run_batch(state):
    c = state["case"]
    b = Batch(state["systems"], state["h"])
    b.set(threads=128, steps_per_launch=31)
    events, system, step = b.advance(0.0, c["steps"], RCEN)
    ends = b.download()
    return dict(x=np.concatenate([e[0] for e in ends]), v=np.concatenate([e[1] for e in ends]),
                **_kept(state, events, system, step))


def _run_adjoint(state):
    c, (x0, v0, yar) = state["case"], state["inputs"]
    xf, vf = mvs_trajectory(x0, v0, yar, state["big"], c["h"], c["steps"], c["every"])
    gx, gv, gy = torch.autograd.grad((xf ** 2).sum(), (x0, v0, yar))
    return dict(x=xf.detach(), v=vf.detach(), gx=gx, gv=gv, gyar=gy)


def _run_hybrid_adjoint(state):
    c, s, (x0, v0, yar) = state["case"], state["system"], state["inputs"]
    nb = s.nbig
    xf, vf = hybrid_trajectory(x0, v0, yar, (*state["big"], s.rcrit[:nb]), s.rcrit[nb:], c["h"], c["steps"], TOL,
                               c["every"])
    gx, gv, gy = torch.autograd.grad((xf ** 2).sum(), (x0, v0, yar))
    return dict(x=xf.detach(), v=vf.detach(), gx=gx, gv=gv, gyar=gy)


RUNS = dict(steps=_run_steps, run=_run_run, output=_run_output, hybrid=_run_hybrid, adaptive=_run_adaptive,
            batch=_run_batch, adjoint=_run_adjoint, hybrid_adjoint=_run_hybrid_adjoint)


def run(state):
    return RUNS[state["case"]["kind"]](state)


# --------------------------------------------------------------------- work
def _particles(case):
    """Particles of all systems of a case."""
    return case["particles"] if case["kind"] != "batch" else int(_sizes(case).sum())


def work(case):
    """Inputs read once and outputs written once; FP64 operations of the map's
    own formulas (a divide or square root is one operation)."""
    kind = case["kind"]
    n, nb, steps = _particles(case), case.get("planets", 4.5), case.get("steps", 1)
    force = 21.0 * nb                 # direct terms of one particle's force
    step = 208.0 + force              # kick, drift, screens, force: 376 with 8 planets
    if kind in ("steps", "run", "batch"):
        return {"bytes": 8.0 * n * 15, "flops": n * steps * step}
    if kind == "output":              # one step, then six drifts and four kicks
        return {"bytes": 8.0 * n * 15, "flops": n * (step + 6 * 120.0 + 4 * force)}
    if kind == "hybrid":
        return {"bytes": 8.0 * n * 16, "flops": n * steps * (step + 12.0 * nb)}
    if kind == "adaptive":            # steps of about a week
        calls = abs(case["days"]) / 7.0 * {"RADAU": 15, "BS": 36, "BS2": 36}[case["method"]]
        return {"bytes": 8.0 * n * 21, "flops": n * calls * (force + 150.0)}
    # forward, the segment again, and about twice a step back through it
    return {"bytes": 8.0 * n * 26, "flops": 4.0 * n * steps * step}


# ------------------------------------------------- the same results in 64 bits
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _dot(a, b):
    return (a * b).sum(-1)


def _stumpff(z):
    """c0 .. c3: the series near zero, the closed forms elsewhere."""
    w = torch.where(z.abs() < 1.0, z, torch.zeros_like(z))
    c2, c3 = torch.zeros_like(w), torch.zeros_like(w)
    for j in range(11, -1, -1):
        c2 = 1.0 / math.factorial(2 * j + 2) - w * c2
        c3 = 1.0 / math.factorial(2 * j + 3) - w * c3
    if bool((z.abs() >= 1.0).any()):
        q = torch.sqrt(z.abs().clamp(min=1.0))
        e2 = torch.where(z > 0, (1 - torch.cos(q)) / q ** 2, (torch.cosh(q.clamp(max=50.0)) - 1) / q ** 2)
        e3 = torch.where(z > 0, (q - torch.sin(q)) / q ** 3, (torch.sinh(q.clamp(max=50.0)) - q) / q ** 3)
        c2 = torch.where(z.abs() < 1.0, c2, e2)
        c3 = torch.where(z.abs() < 1.0, c3, e3)
    return 1.0 - z * c2, 1.0 - z * c3, c2, c3


def _drift(mu, x, v, dt):
    """Two-body motion by dt in universal variables (Laguerre, then Newton)."""
    r0 = torch.sqrt(_dot(x, x))
    u = _dot(x, v)
    alpha = 2.0 * mu / r0 - _dot(v, v)

    def at(s):
        c0, c1, c2, c3 = _stumpff(alpha * s * s)
        g1, g2, g3 = s * c1, s * s * c2, s * s * s * c3
        return r0 * g1 + u * g2 + mu * g3 - dt, r0 * c0 + u * g1 + mu * g2, u * c0 + (mu - alpha * r0) * g1, g1, g2, g3

    with torch.no_grad():
        s = dt / r0
        for k in range(40):
            f, fp, fpp, *_ = at(s)
            ds = 5.0 * f / (fp + torch.sqrt((16.0 * fp * fp - 20.0 * f * fpp).abs()))
            s = s - ds
            if k % 3 == 2 and bool((ds.abs() <= 1e-13 * s.abs()).all()):
                break
    f, fp, *_ = at(s)
    s = s - f / fp
    _, r, _, g1, g2, g3 = at(s)
    a, b = (1.0 - mu * g2 / r0)[..., None], (dt - mu * g3)[..., None]
    c, d = (-mu * g1 / (r * r0))[..., None], (1.0 - mu * g2 / r)[..., None]
    return a * x + b * v, c * x + d * v


def _yarkovsky(x, v, yar):
    r2 = _dot(x, x)
    t = v - (_dot(x, v) / r2)[..., None] * x
    return (yar / (r2 * torch.sqrt(_dot(t, t))))[..., None] * t


def _direct(x, xb, mb):
    a = torch.zeros_like(x)
    for k in range(xb.shape[0]):
        d = x - xb[k]
        a = a - (mb[k] * _dot(d, d) ** -1.5)[..., None] * d
    return a


class _Planets:
    """The planets' part of the symplectic map, in Jacobi coordinates."""

    def __init__(self, m, x, v):
        self.m0, self.m, self.x, self.v = m[0], m[1:], x[1:], v[1:]
        self.inner = torch.cat([torch.zeros_like(m[:1]), torch.cumsum(self.m, 0)[:-1]])   # mass inside each
        self.gm = self.m0 * (self.m0 + self.inner + self.m) / (self.m0 + self.inner)

    def jacobi(self, q):
        c = torch.cumsum(self.m[:, None] * q, 0)
        c = torch.cat([torch.zeros_like(c[:1]), c[:-1]])
        return q - c / (self.m0 + self.inner)[:, None]

    def heliocentric(self, q):
        c = torch.cumsum((self.m / (self.m0 + self.inner + self.m))[:, None] * q, 0)
        return q + torch.cat([torch.zeros_like(c[:1]), c[:-1]])

    def drift(self, dt):
        x, v = _drift(self.gm, self.jacobi(self.x), self.jacobi(self.v), dt)
        self.x, self.v = self.heliocentric(x), self.heliocentric(v)

    def force(self):
        """(accelerations of the planets, the indirect term of a particle's)."""
        x, m, n = self.x, self.m, len(self.m)
        xj = self.jacobi(x)
        r3, rj3 = _dot(x, x) ** -1.5, _dot(xj, xj) ** -1.5
        term = (m * r3)[:, None] * x
        a0 = -term[1:].sum(0)
        sun = self.m0 * (rj3[:, None] * xj - r3[:, None] * x)
        sun[0] = 0.0
        back = (m * self.m0 * rj3 / (self.m0 + self.inner))[:, None] * xj
        back[0] = 0.0
        acc = a0 + sun + torch.cumsum(back, 0)
        for k in range(n):
            others = [q for q in range(n) if q != k]
            if others:
                acc[k] = acc[k] + _direct(x[k], x[others], m[others])
        return acc, a0 - term[0]


def _mvs(m, xb, vb, x, v, yar, h, steps):
    """`steps` steps of the symplectic map: planets and particles, end states."""
    p, mu = _Planets(m, xb, vb), m[0]

    def forces():
        ab, indirect = p.force()
        a = indirect + _direct(x, p.x, p.m)
        return ab, a if yar is None else a + _yarkovsky(x, v, yar)

    ab, a = forces()
    for _ in range(steps):
        p.v, v = p.v + 0.5 * h * ab, v + 0.5 * h * a
        p.drift(h)
        x, v = _drift(mu, x, v, h)
        ab, a = forces()
        p.v, v = p.v + 0.5 * h * ab, v + 0.5 * h * a
    return p, x, v


def _tensors(s):
    t = [torch.tensor(np.array(a), dtype=torch.float64, device=_device())
         for a in (s.m[:s.nbig], s.x[:s.nbig], s.v[:s.nbig], s.x[s.nbig:], s.v[s.nbig:], s.ngf[s.nbig:, 3],
                   s.ngf[s.nbig:, 4])]
    return t


def _all_rows(s, p_x, p_v, x, v):
    """Rows of every body, the central body's as they went in."""
    head = [torch.tensor(np.array(a[:1]), dtype=torch.float64, device=x.device) for a in (s.x, s.v)]
    return torch.cat([head[0], p_x, x]).cpu(), torch.cat([head[1], p_v, v]).cpu()


def _corrector(m, p, x, v, yar, h):
    """The map's coordinates to physical ones (two stages of drifts and kicks)."""
    mu, r10 = m[0], math.sqrt(10.0)
    for ha, hb in ((h * r10 * 0.3, -h * r10 / 72.0), (h * r10 * 0.2, h * r10 / 24.0)):
        for move, sign in ((ha, -1.0), (-2.0 * ha, 1.0), (ha, 0.0)):
            p.drift(move)
            x, v = _drift(mu, x, v, move)
            if sign:
                ab, ind = p.force()
                a = ind + _direct(x, p.x, p.m)
                a = a if yar is None else a + _yarkovsky(x, v, yar)
                p.v, v = p.v + sign * hb * ab, v + sign * hb * a
    return p, x, v


def _ode(m, xb, vb, x, v, beta, yar, days, dust):
    """Planets and particles under gravity and, with `dust`, relativity,
    radiation and Yarkovsky forces, by extrapolated midpoint steps of about two
    days."""
    m0, mb, nb, c = m[0], m[1:], len(m) - 1, LIGHT

    def accel(q, w):
        qb, r2 = q[:nb], _dot(q, q)
        r = torch.sqrt(r2)
        a = -(mb[:, None] * qb * (r2[:nb] ** -1.5)[:, None]).sum(0) + torch.zeros_like(q)
        for k in range(nb):
            d = q - qb[k]
            d2 = _dot(d, d)
            d2[k] = 1.0
            a = a - (mb[k] * d2 ** -1.5)[:, None] * d
        r3 = m0 / (r * r2)
        a = a - r3[:, None] * q
        if not dust:
            return a
        rv, v2 = _dot(q, w), _dot(w, w)
        a = a + (r3 / c ** 2)[:, None] * ((4 * m0 / r - v2)[:, None] * q + (4 * rv)[:, None] * w)
        qs, ws, rs = q[nb:], w[nb:], r[nb:]
        k = (K2 * beta / rs ** 2)[:, None]
        pr = k * ((1 - 1.3 * rv[nb:] / rs / c)[:, None] * qs / rs[:, None] - 1.3 * ws / c)
        return torch.cat([a[:nb], a[nb:] + pr + _yarkovsky(qs, ws, yar)])

    q, w = torch.cat([xb[1:], x]), torch.cat([vb[1:], v])
    count = max(1, math.ceil(abs(days) / 2.0))
    big, levels = days / count, (2, 4, 6, 8, 10, 12, 14)
    for _ in range(count):
        rows, start = [], accel(q, w)
        for k, n in enumerate(levels):
            hh = big / n
            qa, wa, qc, wc = q, w, q + hh * w, w + hh * start
            for _ in range(n - 1):
                a = accel(qc, wc)
                qa, wa, qc, wc = qc, wc, qa + 2 * hh * wc, wa + 2 * hh * a
            a = accel(qc, wc)
            row = [(0.5 * (qa + qc + hh * wc) - q, 0.5 * (wa + wc + hh * a) - w)]
            for j in range(1, k + 1):
                f = (levels[k] / levels[k - j]) ** 2 - 1.0
                row.append(tuple(row[j - 1][e] + (row[j - 1][e] - rows[k - 1][j - 1][e]) / f for e in (0, 1)))
            rows.append(row)
        q, w = q + rows[-1][-1][0], w + rows[-1][-1][1]
    return q[:nb], w[:nb], q[nb:], w[nb:]


def _energy(m, xb, vb):
    """Energy and angular momentum of the massive bodies about their centre of
    mass (heliocentric rows in)."""
    tot = m.sum()
    x = torch.cat([torch.zeros_like(xb[:1]), xb[1:]])
    v = torch.cat([torch.zeros_like(vb[:1]), vb[1:]])
    x, v = x - (m[:, None] * x).sum(0) / tot, v - (m[:, None] * v).sum(0) / tot
    e = (0.5 * m * _dot(v, v)).sum()
    for i in range(len(m)):
        for j in range(i):
            d = x[i] - x[j]
            e = e - m[i] * m[j] / torch.sqrt(_dot(d, d))
    ang = (m[:, None] * torch.linalg.cross(x, v)).sum(0)
    return float(e), float(torch.sqrt(_dot(ang, ang)))


def exact(case, seed):
    kind = case["kind"]
    if kind in ("hybrid", "hybrid_adjoint", "batch"):
        return None   # thousands of small systems, or subsystems picked by a screen: minutes in torch
    if kind == "run" and case["steps"] > 100:
        return None   # encounters have multiplied the last bit of the map's own rounding into the first by then
    if kind == "adaptive" and case["particles"] * abs(case["days"]) > 4e7:
        return None
    s = _system(case, seed)
    m, xb, vb, x, v, beta, yar = _tensors(s)
    if kind == "adaptive":
        with torch.no_grad():
            rows = _all_rows(s, *_ode(m, xb, vb, x, v, beta, yar, case["days"], s.pn != 0))
        return dict(x=rows[0], v=rows[1])
    if kind == "adjoint":
        if case["steps"] <= 300 and case["steps"] * case["particles"] <= 1_000_000:   # some seconds at most
            ends, grads = [], []
            for k in range(0, x.shape[0], 4000):
                part = [q[k:k + 4000].clone().requires_grad_() for q in (x, v, yar)]
                _, xf, vf = _mvs(m, xb, vb, *part, case["h"], case["steps"])
                grads.append(torch.autograd.grad((xf ** 2).sum(), part))
                ends.append((xf.detach(), vf.detach()))
            got = [torch.cat([e[q] for e in ends]) for q in (0, 1)] + [torch.cat([g[q] for g in grads]) for q in range(3)]
            return dict(zip(("x", "v", "gx", "gv", "gyar"), got))
        with torch.no_grad():
            _, x, v = _mvs(m, xb, vb, x, v, yar, case["h"], case["steps"])
        return dict(x=x, v=v)
    with torch.no_grad():
        p, x, v = _mvs(m, xb, vb, x, v, yar if case["yar"] else None, case["h"], case.get("steps", 1))
        if kind == "output":
            p, x, v = _corrector(m, p, x, v, yar if case["yar"] else None, case["h"])
    rows = _all_rows(s, p.x, p.v, x, v)
    if kind == "output":
        nb = s.nbig
        e, l2 = _energy(m, rows[0][:nb].to(m.device), rows[1][:nb].to(m.device))
        return dict(x=rows[0], v=rows[1], energy=e, l2=l2)
    return dict(x=rows[0], v=rows[1])
