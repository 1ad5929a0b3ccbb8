"""The work that the framework does for its users, as cases that can be timed.

Every case goes through the public ``Domain`` API (and the sweep and adjoint
modules on top of it), as a program that runs explicit SPH steps does:

* ``upset``   a cylinder upset between two velocity zones, the workload of the
              benchmark and of the parity tests: the plain FP64 and the mixed
              form, elastic and yielding, bilinear or Johnson-Cook with
              conduction and plastic heating, kick-drift or leapfrog, with or
              without the tensile-instability term;
* ``contact`` the same cylinder pressed by a rigid plane with friction;
* ``sweep``   uneven Johnson-Cook specimens stepped together in one domain;
* ``search``  positions written by the program, then the neighbour search;
* ``adjoint`` a reaction-force loss and its gradient by the adjoint.

A stepping pass rewinds the domain to a checkpoint taken after the first
steps, runs ``steps`` steps and reads the fields: what a program does between
two outputs (the reference's inputs write every ~18 to ~2000 steps; a pass
here takes 4 to 50).  The plain form's fields are returned in FP64.  The mixed
form sums its pairs in FP32 and states its accuracy as 1e-4, so a program
that runs it keeps its snapshots in FP32: its fields are returned like that.

Sizes and physical constants are the repository's own: configurations 1 to 3,
the sweep's specimens, the adjoint's cylinder and the reference decks' 4k to
40k particles, besides sizes between them.
"""
import math

import numpy as np
import torch

import weldform_gb300 as wf
from weldform_gb300 import adjoint, batch, configs

MIXED, FP64 = "mixed", "fp64"
STEEL = configs.Steel()


def _upset(name, form, dx_mm, steps, warm, v=-1.0, jc=False, leapfrog=False, ti=False, R_mm=10.0, L_mm=30.0):
    c = {"kind": "upset", "form": form, "R_mm": R_mm, "L_mm": L_mm, "dx_mm": dx_mm, "v": v, "jc": jc,
         "leapfrog": leapfrog, "ti": ti, "warm": warm, "steps": steps}
    return dict(c, name=name) if name else c


def _contact(name, form, dx_mm, steps, warm, v, friction, stiffness, jc=True, ti=False, R_mm=10.0, L_mm=30.0):
    c = {"kind": "contact", "form": form, "R_mm": R_mm, "L_mm": L_mm, "dx_mm": dx_mm, "v": v, "friction": friction,
         "stiffness": stiffness, "jc": jc, "ti": ti, "warm": warm, "steps": steps}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the benchmark's cylinder (982,072 particles), elastic: no search inside the pass
        _upset("upset_982k_mixed", MIXED, 0.2112, 20, 3),
        # the same cylinder yielding: a neighbour search every 5 steps
        _upset("upset_982k_mixed_yield", MIXED, 0.2112, 20, 25, v=-20.0),
        # penalty-contact press with Johnson-Cook hardening, conduction and plastic heating (1,150,200 particles)
        _contact("contact_1150k_mixed", MIXED, 0.2, 10, 6, -20.0, 0.2, "area"),
        # 36 uneven specimens in one domain, each with its own rebuild schedule: a parameter study
        {"name": "sweep_36_mixed", "kind": "sweep", "form": MIXED, "specimens": 36, "dx_mm": 0.5, "warm": 12, "steps": 12},
        # a middle size at an odd count, thermal and yielding: a component study on the mixed form
        _upset("upset_79k_mixed_thermal", MIXED, 0.487, 20, 20, v=-20.0, jc=True, R_mm=9.7, L_mm=30.9),
        # the JSON driver's leapfrog solver with its default tensile-instability term, at the decks' size
        _upset("upset_31k_mixed_leapfrog", MIXED, 0.66, 30, 10, v=-5.0, leapfrog=True, ti=True),
        # a reference deck: rigid-plane press, Wang's stiffness with friction, tensile instability on
        _contact("contact_12k_mixed", MIXED, 0.92, 30, 10, -1.0, 0.6, "wang", jc=False, ti=True),
        # the smallest configuration, 8,004 particles: a step is a few launches of a few microseconds
        _upset("upset_8k_mixed", MIXED, 1.0, 50, 3),
        # the smallest configuration in the plain FP64 form, yielding
        _upset("upset_8k_fp64", FP64, 1.0, 20, 20, v=-20.0),
        # the plain FP64 form at the middle size of its parity and accuracy runs (240,300 particles)
        _upset("upset_240k_fp64", FP64, 0.3353, 5, 3),
        # positions written by the program (restart, remap), then a full search
        {"name": "search_240k", "kind": "search", "form": MIXED, "R_mm": 10.0, "L_mm": 30.0, "dx_mm": 0.3353},
        # calibration: loss and gradient of a reaction-force curve with respect to the material parameters
        {"name": "adjoint_17k", "kind": "adjoint", "form": FP64, "dx_mm": 0.8, "v": -20.0, "steps": 40, "every": 10,
         "chk": 20},
    ]


def draw(rng):
    """One more case of the same kinds; sizes spread over their logarithm."""
    def dx_for(n, R_mm, L_mm):
        return round((math.pi * R_mm * R_mm * L_mm / n) ** (1.0 / 3.0), 4)

    def count(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    kind = rng.choice(["upset", "upset", "upset", "upset", "contact", "contact", "sweep", "search", "adjoint"])
    R = round(rng.uniform(7.0, 10.0), 2)
    L = round(R * rng.uniform(2.0, 3.0), 2)
    if kind == "upset":
        form = rng.choice([MIXED, MIXED, FP64])
        n = count(5e3, 1.0e6) if form == MIXED else count(5e3, 2.4e5)
        steps = max(4, min(40, int(1.5e7 / n))) if form == MIXED else max(3, min(20, int(1.0e6 / n)))
        leapfrog = rng.random() < 0.25
        return _upset(None, form, dx_for(n, R, L), steps, rng.randint(3, 20), v=rng.choice([-1.0, -5.0, -20.0]),
                      jc=rng.random() < 0.4, leapfrog=leapfrog, ti=rng.random() < 0.3, R_mm=R, L_mm=L)
    if kind == "contact":
        form = rng.choice([MIXED, MIXED, FP64])
        n = count(6e3, 1.0e6) if form == MIXED else count(6e3, 1.2e5)
        steps = max(4, min(30, int(8e6 / n))) if form == MIXED else max(3, min(15, int(6e5 / n)))
        return _contact(None, form, dx_for(n, R, L), steps, rng.randint(3, 10), rng.choice([-1.0, -20.0]),
                        rng.choice([0.0, 0.2]), rng.choice(["area", "penalty"]), jc=rng.random() < 0.6, R_mm=R, L_mm=L)
    if kind == "sweep":
        return {"kind": "sweep", "form": MIXED, "specimens": rng.randint(3, 40), "dx_mm": 0.5,
                "warm": rng.randint(3, 15), "steps": rng.randint(4, 12)}
    if kind == "search":
        return {"kind": "search", "form": rng.choice([MIXED, FP64]), "R_mm": R, "L_mm": L,
                "dx_mm": dx_for(count(1e4, 5e5), R, L)}
    return {"kind": "adjoint", "form": FP64, "dx_mm": round(rng.uniform(0.8, 1.2), 3), "v": -20.0,
            "steps": 10 * rng.randint(2, 4), "every": 10, "chk": rng.choice([10, 20])}


# ---------------------------------------------------------------- inputs
def _jitter(n, dx, seed):
    """Position offsets of a packed specimen: +-1e-3 of the spacing."""
    return np.random.default_rng(int(seed)).uniform(-1.0, 1.0, (n, 3)) * (1e-3 * dx)


def _specimens(case, seed):
    """Radius 4 to 8 mm, L/D 1 to 2, Johnson-Cook constants within +-20 %, punch speed 0.5 to 5 m/s."""
    sizes = np.random.default_rng(case["specimens"])  # sizes belong to the case, values to the seed
    rng = np.random.default_rng(int(seed))
    out = []
    A, B, n, C, e0, m, Tm, Tt = STEEL.jc
    for _ in range(case["specimens"]):
        R = float(sizes.uniform(0.004, 0.008))
        length = float(2 * R * sizes.uniform(1.0, 2.0))
        f = rng.uniform(0.8, 1.2, size=5)
        out.append(batch.Specimen(R=R, L=length, v_punch=-float(rng.uniform(0.5, 5.0)),
                                  jc=(A * f[0], B * f[1], n * f[2], C * f[3], e0, m * f[4], Tm, Tt)))
    return out


def _fields(case):
    f = [("Displacement", 3), ("v", 3), ("Sigma", 9), ("Density", 1), ("pl_strain", 1)]
    if case["kind"] in ("upset", "contact") and case["jc"]:
        f.append(("T", 1))
    return f


class State:
    def __init__(self, case, dom, n):
        self.case, self.dom, self.n = case, dom, n
        self.out = {}

    def buffers(self):
        """Host buffers that the program keeps for its fields: page-locked, as an asynchronous reader wants them."""
        for name, comps in _fields(self.case):
            shape = (self.n, comps) if comps > 1 else (self.n,)
            buf = torch.empty(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())
            kept = buf if self.case["form"] == FP64 else torch.empty(shape, dtype=torch.float32)
            self.out[name] = (buf, buf.numpy(), kept)


def _domain(case):
    dom = wf.Domain()
    dom.set("precision", wf.PRECISION_MIXED if case["form"] == MIXED else wf.PRECISION_FP64)
    return dom


def prepare(case, seed):
    kind = case["kind"]
    dom = _domain(case)
    if kind == "adjoint":
        cc = adjoint.ContactCase(R=0.010, L=0.030, dx=case["dx_mm"] * 1e-3, v_punch=case["v"], seed=int(seed))
        adjoint.build(dom, cc, cc.nominal())
        dom.prepare(cc.dt)
        dom.step(10)
        dom.checkpoint_save(0)
        s = State(case, dom, dom.particle_count)
        # the curve to be met: measured forces near the model's own
        s.target = np.random.default_rng(int(seed)).uniform(-2e4, -1e4, case["steps"] // case["every"])
        return s
    if kind == "sweep":
        specs = _specimens(case, seed)
        sw = batch.build_sweep(dom, specs, dx=case["dx_mm"] * 1e-3, jitter_amp=0.0)
        x = dom.get_array("x")
        for k, (a, b) in enumerate(sw.ranges):
            x[a:b] += _jitter(b - a, sw.dx, int(seed) + k)
        dom.set_array("x", x)
        dt = sw.dt
    else:
        geo = dict(R=case["R_mm"] * 1e-3, L=case["L_mm"] * 1e-3, dx=case["dx_mm"] * 1e-3, jitter_amp=0.0)
        if kind == "contact":
            c = configs.contact_upsetting(dom, v_punch=case["v"], friction=case["friction"],
                                          stiffness=case["stiffness"], thermal=case["jc"], **geo)
        else:
            jc = kind == "upset" and case["jc"]
            c = configs.cylinder_upsetting(dom, v_top=case["v"] if kind == "upset" else -1.0,
                                           model=wf.JOHNSON_COOK if jc else wf.BILINEAR, thermal=jc, **geo)
        dt = c.dt
        if kind in ("upset", "contact") and case["ti"]:
            dom.set_particles("TI", 0.3)
            dom.set_particles("TIn", 4.0)
            dom.set_particles("TIInitDist", c.dx)
        x = dom.get_array("x")
        x[:c.n] += _jitter(c.n, c.dx, seed)
        dom.set_array("x", x)
        if kind == "upset" and case["leapfrog"]:
            dom.set("integrator", 1)
    dom.prepare(dt)
    if kind == "search":
        dom.step(1)
        s = State(case, dom, dom.particle_count)
        # positions of a restart: the body upset by some percent, each particle off its place by up to 5 % of the spacing
        rng = np.random.default_rng(int(seed) + 1)
        squeeze = 1.0 + rng.uniform([-0.01, -0.01, -0.05], [0.01, 0.01, -0.01])
        s.x = torch.from_numpy(x * squeeze + _jitter(len(x), 50 * c.dx, int(seed) + 2)).pin_memory().numpy()
        return s
    dom.step(case["warm"])
    dom.checkpoint_save(0)
    s = State(case, dom, dom.particle_count)
    s.buffers()
    return s


# ---------------------------------------------------------------- one pass
def run(s):
    dom, case = s.dom, s.case
    if case["kind"] == "search":
        dom.set_array("x", s.x)
        dom.neighbour_search()
        return {"Nb": dom.get_array("Nb")}
    dom.checkpoint_restore(0)
    if case["kind"] == "adjoint":
        r = dom.adjoint_reaction_loss(case["steps"], case["every"], s.target, checkpoint_every=case["chk"])
        return {"loss": float(r["loss"]), "curve": r["curve"], "grad": r["grad"]}
    dom.step(case["steps"])
    res = {}
    for name, (buf, arr, kept) in s.out.items():
        dom.get_array(name, out=arr)
        if kept is not buf:
            kept.copy_(buf)
        res[name] = kept
    if case["kind"] == "contact":
        force = torch.from_numpy(dom.contact_force(0))
        res["force"] = force if case["form"] == FP64 else force.to(torch.float32)
    return res


# ---------------------------------------------------------------- what a pass cannot do without
def _count(case):
    if case["kind"] == "sweep":
        return batch.sweep_particles(_specimens(case, 0), case["dx_mm"] * 1e-3)
    R, L = (0.010, 0.030) if case["kind"] == "adjoint" else (case["R_mm"] * 1e-3, case["L_mm"] * 1e-3)
    return configs.cylinder_count(R, L, case["dx_mm"] * 1e-3)


# Per particle and step: x, v, Displacement (9), density, deviatoric stress,
# strain, plastic strain (18), plastic strain scalar and flow stress, read and
# written once in FP64 (30 values each way, 480 B), and the particle's ~55
# neighbour indices; the three pair sums at ~205 operations a pair.
NNZ, STATE_BYTES, PAIR_OPS, PARTICLE_OPS = 54.6, 480.0, 205.0, 300.0


def work(case):
    n = float(_count(case))
    step = {"bytes": n * (STATE_BYTES + 4 * NNZ), "flops": n * (NNZ * PAIR_OPS + PARTICLE_OPS)}
    if case["kind"] == "search":  # positions in, rows and their lengths out; a distance test per row entry
        return {"bytes": n * (24.0 + 4 * NNZ + 4.0), "flops": n * NNZ * 9.0}
    if case["kind"] == "adjoint":  # forward, recompute, and a reverse step of about twice a forward one
        return {k: 4.0 * case["steps"] * v for k, v in step.items()}
    size = 8.0 if case["form"] == FP64 else 4.0
    out = size * n * sum(c for _, c in _fields(case))
    return {"bytes": case["steps"] * step["bytes"] + out, "flops": case["steps"] * step["flops"]}


# ---------------------------------------------------------------- the same in 64 bits, from the equations
def _lattice(R, L, dx):
    """The packed cylinder: rows along x in each y row of each z layer."""
    r = dx / 2

    def half(inc):
        c, yp, xp = 1, r, r + (inc - 1) * 2. * r
        while math.sqrt(yp * yp + xp * xp) <= R - r:
            yp += 2. * r
            c += 1
        return c - 1

    nxy = half(1)
    rows, yp, inc, sign = [], -r - (2. * r * (nxy - 1)), nxy, -1
    for _ in range(2 * nxy):
        nx = half(inc)
        x = np.cumsum(np.r_[-r - (2. * r * (nx - 1)), np.full(2 * nx - 1, 2. * r)])
        rows.append(np.stack([x, np.full(2 * nx, yp)], 1))
        yp += 2. * r
        inc += sign
        if inc < 1:
            inc, sign = 1, 1
    layer = np.concatenate(rows)
    out, zp = [], r
    while zp <= L - r:
        out.append(np.c_[layer, np.full(len(layer), zp)])
        zp += 2. * r
    return np.concatenate(out)


def _pairs(x, R):
    """Neighbours within R as a padded table [n, width] (own index where there is none) in ascending order."""
    n, dev = x.shape[0], x.device
    lo = x.min(0).values - 2 * R
    q = ((x - lo) / R).floor().long()
    dims = (q.max(0).values + 3).tolist()
    key = (q[:, 0] * dims[1] + q[:, 1]) * dims[2] + q[:, 2]
    order = torch.argsort(key, stable=True)
    cells = dims[0] * dims[1] * dims[2]
    cnt = torch.bincount(key, minlength=cells)
    start = torch.cumsum(cnt, 0) - cnt
    width = int(cnt.max())
    slot = torch.arange(n, device=dev) - start[key[order]]
    table = torch.full((cells, width), -1, dtype=torch.long, device=dev)
    table[key[order], slot] = order
    me, other = [], []
    ids = torch.arange(n, device=dev)
    for a in (-1, 0, 1):
        for b in (-1, 0, 1):
            for c in (-1, 0, 1):
                cand = table[key + (a * dims[1] + b) * dims[2] + c]
                d = x[:, None, :] - x[cand.clamp(min=0)]
                ok = (cand >= 0) & (cand != ids[:, None]) & ((d * d).sum(2) <= R * R)
                i, k = ok.nonzero(as_tuple=True)
                me.append(i)
                other.append(cand[i, k])
    i, j = torch.cat(me), torch.cat(other)
    i, j = (t[torch.argsort(i * n + j)] for t in (i, j))
    deg = torch.bincount(i, minlength=n)
    at = torch.arange(i.numel(), device=dev) - (torch.cumsum(deg, 0) - deg)[i]
    nb = ids[:, None].repeat(1, int(deg.max()))
    nb[i, at] = j
    return nb


class _Exact:
    """The explicit step on one body, every value in FP64: cubic spline,
    Monaghan viscosity, Jaumann rate, radial return, two velocity zones."""

    def __init__(self, x, h, mass, dt, z_lo, z_hi, v_top, jc=None, thermal=False, leapfrog=False, ti=0.0, ti_dist=0.0):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.x = torch.as_tensor(x, dtype=torch.float64, device=dev)
        n = self.x.shape[0]
        z = lambda *s: torch.zeros(*s, dtype=torch.float64, device=dev)  # noqa: E731
        self.n, self.h, self.m, self.dt = n, h, mass, dt
        self.fix, self.top, self.v_top = self.x[:, 2] <= z_lo, self.x[:, 2] >= z_hi, v_top
        self.fix = self.fix & ~self.top
        self.jc, self.thermal, self.leapfrog, self.ti, self.ti_dist = jc, thermal, leapfrog, ti, ti_dist
        self.v, self.u, self.rho = z(n, 3), z(n, 3), torch.full_like(self.x[:, 0], STEEL.rho)
        self.tau, self.sig, self.pl, self.dpl = z(n, 3, 3), z(n, 3, 3), z(n), z(n)
        self.epli = z(n, 3, 3)
        self.T, self.dTdt, self.qpl = torch.full_like(self.rho, STEEL.T0), z(n), z(n)
        Th = (STEEL.T0 - jc[7]) / (jc[6] - jc[7]) if jc else 0.0
        self.sy = torch.full_like(self.rho, (jc[0] + jc[1] * 0.0 ** jc[2]) * (1.0 - Th ** jc[5]) if jc else STEEL.sy0)
        self.Ep = 0.0 if jc else STEEL.E * STEEL.Et / (STEEL.E - STEEL.Et)
        self.first, self.yielding, self.ts, self.cleared = True, False, 0, True

    def bc(self, v, a=None):
        v[self.fix] = 0.0
        v[self.top] = torch.tensor([0.0, 0.0, self.v_top], dtype=torch.float64, device=v.device)
        if a is not None:
            a[self.fix | self.top] = 0.0

    def gk(self, d):
        """GradKernel and distances of row differences d; 0 for the padding (own index)."""
        r = torch.linalg.vector_norm(d, dim=2)
        q = r / self.h
        C = 1.0 / (math.pi * self.h ** 4)
        g = torch.where(q < 1.0, C / self.h * (-3.0 + 2.25 * q),
                        torch.where(q < 2.0, -0.75 * C * (2.0 - q) ** 2 / r.clamp(min=1e-300), torch.zeros_like(q)))
        return torch.where(r == 0.0, torch.zeros_like(g), g), r

    def rows(self):
        size = max(1, (1 << 25) // self.nb.shape[1])
        for a in range(0, self.n, size):
            yield slice(a, min(self.n, a + size)), self.nb[a:a + size]

    def step(self):
        mx = float(self.pl.max())
        search = False
        if mx > 1e-6 and not self.yielding:
            search, self.yielding = True, True
        elif (mx > 1e-6 or self.first) and self.ts == 0 and self.cleared:
            search = True
        if search:
            self.cleared = False
            self.nb = _pairs(self.x, 2.0 * self.h)
        dt, m, h = self.dt, self.m, self.h
        S = self.sig / (self.rho ** 2)[:, None, None]
        if self.ti > 0.0:
            parts = [torch.linalg.eigh(t) for t in self.sig.split(8192)]  # in batches that the solver takes
            ev, V = torch.cat([p.eigenvalues for p in parts]), torch.cat([p.eigenvectors for p in parts])
            f = torch.where(ev > 0.0, -self.ti / (self.rho ** 2)[:, None] * ev, torch.zeros_like(ev))
            tir = (V * f[:, None, :]) @ V.transpose(1, 2)
            q0 = self.ti_dist / h
            w0 = 1.0 - 1.5 * q0 ** 2 + 0.75 * q0 ** 3 if q0 < 1.0 else 0.25 * max(0.0, 2.0 - q0) ** 3
        a = torch.zeros_like(self.x)
        eye = torch.eye(3, dtype=torch.float64, device=self.x.device)
        for s, nb in self.rows():
            d = self.x[s, None, :] - self.x[nb]
            g, r = self.gk(d)
            dvx = ((self.v[s, None, :] - self.v[nb]) * d).sum(2)
            mu = h * dvx / (r * r + 0.01 * h * h)
            pi = torch.where(dvx < 0.0, STEEL.Cs * mu / (0.5 * (self.rho[s, None] + self.rho[nb])), torch.zeros_like(mu))
            Sp = S[s, None] + S[nb] + pi[:, :, None, None] * eye
            if self.ti > 0.0:
                q = r / h
                w = torch.where(q < 1.0, 1.0 - 1.5 * q ** 2 + 0.75 * q ** 3, 0.25 * (2.0 - q).clamp(min=0.0) ** 3)
                Sp = Sp + ((w / w0) ** 4)[:, :, None, None] * (tir[s, None] + tir[nb])
            a[s] = ((m * g)[:, :, None] * (Sp @ d[:, :, :, None])[..., 0]).sum(1)
        v = self.v
        if self.leapfrog:
            if self.first:
                v = v - a * 0.5 * dt
            self.bc(v, a)
            v = v + a * dt
        else:
            self.bc(v, a)
            v = v + a * 0.5 * dt
        self.bc(v, a)
        V = m / self.rho
        drho = torch.zeros_like(self.rho)
        for s, nb in self.rows():
            d = self.x[s, None, :] - self.x[nb]
            g, _ = self.gk(d)
            drho[s] = self.rho[s] * (V[nb] * g * ((v[s, None, :] - v[nb]) * d).sum(2)).sum(1)
        self.rho = self.rho + dt * drho
        self.x, self.u = self.x + v * dt, self.u + v * dt
        v = v if self.leapfrog else v + a * dt / 2.0
        self.bc(v)
        self.v = v
        if self.thermal:
            self.T = self.T + dt * self.dTdt
        V = m / self.rho
        ids = torch.arange(self.n, device=self.x.device)
        Lg = torch.zeros_like(self.tau)
        cond = torch.zeros_like(self.rho)
        for s, nb in self.rows():
            d = self.x[s, None, :] - self.x[nb]
            g, _ = self.gk(d)
            w = (V[nb] * -g)[:, :, None] * (self.v[s, None, :] - self.v[nb])
            Lg[s] = w.transpose(1, 2) @ d
            if self.thermal:
                Vp = torch.where(nb > ids[s, None], V[nb], V[s, None])
                cond[s] = (Vp * 4.0 * (STEEL.k_T / 2.0) * (self.T[s, None] - self.T[nb]) * g).sum(1)
        self.stress(0.5 * (Lg + Lg.transpose(1, 2)), 0.5 * (Lg - Lg.transpose(1, 2)), cond)
        self.first = False
        if mx > 1e-6:
            if self.ts == 4:
                self.cleared = True
            self.ts = (self.ts + 1) % 5

    def stress(self, D, W, cond):
        dt, G = self.dt, STEEL.G
        eye = torch.eye(3, dtype=torch.float64, device=D.device)
        p = STEEL.Cs ** 2 * (self.rho - STEEL.rho)
        tr = D.diagonal(dim1=1, dim2=2).sum(1)
        tau = self.tau + dt * (2.0 * G * (D - tr[:, None, None] / 3.0 * eye) + self.tau @ W.transpose(1, 2) + W @ self.tau)
        d0, d1, d2 = D[:, 0, 0], D[:, 1, 1], D[:, 2, 2]
        rate = torch.sqrt(0.5 * ((d0 - d1) ** 2 + (d1 - d2) ** 2 + (d2 - d0) ** 2) +
                          3.0 * (D[:, 0, 1] ** 2 + D[:, 1, 2] ** 2 + D[:, 0, 2] ** 2))
        trial = torch.sqrt(1.5 * (tau * tau).sum((1, 2)))
        sc = torch.where(trial > 0.0, (self.sy / trial.clamp(min=1e-300)).clamp(max=1.0), torch.ones_like(trial))
        tau = tau * sc[:, None, None]
        if self.jc:
            A, B, n, C, e0, mm, Tm, Tt = self.jc
            # the step's flow stress reads the temperature before this step's increment
            f = torch.where(rate > e0, 1.0 + C * torch.log(rate.clamp(min=1e-300) / e0), torch.ones_like(rate))
            T = self.T - dt * self.dTdt if self.thermal else self.T
            Th = (T - Tt) / (Tm - Tt)
            self.sy = (A + B * self.pl ** n) * f * (1.0 - Th ** mm)
        dep = torch.where(trial > self.sy, (trial - self.sy) / (3.0 * G + self.Ep), torch.zeros_like(trial))
        hit = dep > 0.0
        self.pl = self.pl + dep
        self.dpl = torch.where(hit, dep, self.dpl)
        if not self.jc:
            self.sy = self.sy + dep * self.Ep
        self.tau, self.sig = tau, tau - p[:, None, None] * eye
        tot = self.sig.diagonal(dim1=1, dim2=2).sum(1)
        inc = (dep / self.sy)[:, None, None] * 1.5 * (self.sig - (tot / 3.0)[:, None, None] * eye)
        self.epli = torch.where(hit[:, None, None], inc, self.epli)
        if self.thermal:
            q = (self.sig * self.epli).sum((1, 2)) / dt
            self.qpl = torch.where(self.dpl > 0.0, q, self.qpl)
            self.dTdt = (cond + 0.9 * self.qpl) / (self.rho * STEEL.cp_T)


def _run_exact(e, steps):
    for _ in range(steps):
        e.step()
    out = {"Displacement": e.u, "v": e.v, "Sigma": e.sig.reshape(-1, 9), "Density": e.rho, "pl_strain": e.pl, "T": e.T}
    return {k: t.cpu() for k, t in out.items()}


def exact(case, seed):
    """None for the kinds whose outputs are not a closed sequence of these
    equations: the contact pass (its searches decide by geometry), the
    gradient, and the search's whole numbers."""
    kind = case["kind"]
    if kind not in ("upset", "sweep"):
        return None
    dx = case["dx_mm"] * 1e-3
    h = 1.2 * dx
    dt = 0.4 * h / STEEL.Cs
    steps = case["warm"] + case["steps"]
    if kind == "upset":
        R, L = case["R_mm"] * 1e-3, case["L_mm"] * 1e-3
        x = _lattice(R, L, dx)
        x = x + _jitter(len(x), dx, seed)
        # zones are assigned on the lattice, before the program jitters it
        z0 = _lattice_z(L, dx)
        z_lo, z_hi = _between(z0, 2 * dx, True), _between(z0, L - 3 * dx, False)
        e = _Exact(x, h, math.pi * R * R * L * STEEL.rho / len(x), dt, z_lo, z_hi, case["v"],
                   jc=STEEL.jc if case["jc"] else None, thermal=case["jc"], leapfrog=case["leapfrog"],
                   ti=0.3 if case["ti"] else 0.0, ti_dist=dx)
        out = _run_exact(e, steps)
        return {name: out[name] for name, _ in _fields(case)}
    if _count(case) * steps > 3e7:
        return None
    parts = []
    for k, s in enumerate(_specimens(case, seed)):
        x = _lattice(s.R, s.L, dx)
        x = x + _jitter(len(x), dx, int(seed) + k)
        z0 = _lattice_z(s.L, dx)
        e = _Exact(x, h, math.pi * s.R * s.R * s.L * STEEL.rho / len(x), dt, _between(z0, 2 * dx, True),
                   _between(z0, s.L - 3 * dx, False), s.v_punch, jc=s.jc)
        parts.append(_run_exact(e, steps))
    return {name: torch.cat([p[name] for p in parts]) for name, _ in _fields(case)}


def _lattice_z(L, dx):
    z, zp = [], dx / 2
    while zp <= L - dx / 2:
        z.append(zp)
        zp += dx
    return np.array(z)


def _between(z, bound, below):
    """A height between the layers that the bound takes in and the others."""
    taken = z[z <= bound] if below else z[z >= bound]
    half = 0.5 * (z[1] - z[0])
    return float(taken.max() + half) if below else float(taken.min() - half)
