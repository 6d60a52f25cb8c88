"""The calls whose speed this library is held to, as a user's program makes them.

A case is a dict of plain values; prepare() makes the solver (or batch) a program holds before
the call, from a config whose droplet, interface and fluids are drawn from the seed; run() is
one pass: some steps of the flow and the state read back, or one gradient.

kinds
  steps    solve(n), then c and the velocity into device buffers: a long run between two outputs
  monitor  n times solve_monitored(1): a run that watches mass and kinetic energy at every step
  loop     the reference's main loop: n times NSAllen.solve(), then DataArray.updateHost()
  batch    many 2D cases in one Batch: solve(n), every case's c, velocity and monitors
  adjoint  gradient of the centroid objective after n steps (forward run and reverse sweep)
"""
import math
import os
import tempfile

import numpy as np
import torch

import clip_b200 as cb

GRAVITY = 1e-6


# ---------------------------------------------------------------- the cases
def _case(name, kind, flow, size, precision, steps, sides="pwp", tuned=False, count=0):
    """sides: one letter per axis, p periodic, w wall; 'jet' a velocity inlet at y+ with a
    free outflow at y- and periodic x and z.  tuned: the program calls autotune() first."""
    nx, ny, nz = size
    return dict(name=name, kind=kind, flow=flow, nx=nx, ny=ny, nz=nz, precision=precision, steps=steps, sides=sides,
                tuned=tuned, count=count)


def listed():
    return [
        # the benchmark's production run: rising bubble, launch shape tuned once
        _case("bubble3d_large_fp32", "steps", "bubble", (256, 512, 256), "fp32", 20, tuned=True),
        # the half-size bubble in the reference's precision, launched as created
        _case("bubble3d_fp64", "steps", "bubble", (128, 256, 128), "fp64", 6),
        # the same in half-precision storage, for runs that must hold more nodes
        _case("bubble3d_fp16_tuned", "steps", "bubble", (128, 256, 128), "fp16", 20, tuned=True),
        # a run that reports at every step
        _case("bubble3d_monitored_fp32", "monitor", "bubble", (128, 256, 128), "fp32", 10, tuned=True),
        # a small 3D study, launched as created
        _case("bubble3d_small_fp32", "steps", "bubble", (64, 96, 64), "fp32", 20),
        # a closed box of sizes that divide by nothing
        _case("drop3d_ragged_box_fp32", "steps", "drop", (97, 131, 83), "fp32", 20, sides="www"),
        # an injected jet: velocity inlet and free outflow
        _case("jet3d_fp32", "steps", "jet", (64, 160, 64), "fp32", 20, sides="jet"),
        # Rayleigh-Taylor instability: a long thin 2D run, in both precisions
        _case("rti2d_fp32", "steps", "RTI", (256, 1024, 1), "fp32", 100, sides="pw"),
        _case("rti2d_ragged_fp64", "steps", "RTI", (201, 777, 1), "fp64", 50, sides="pw"),
        # the smallest case of the repository in the reference-shaped loop
        _case("drop2d_loop_fp64", "loop", "drop", (64, 128, 1), "fp64", 10, sides="pw"),
        # a parameter study: many small 2D cases at once
        _case("batch512_fp32", "batch", "mixed", (256, 512, 1), "fp32", 60, sides="pw", tuned=True, count=512),
        # the gradient of an inverse problem on the 256 x 256 drop
        _case("adjoint2d_fp64", "adjoint", "drop", (256, 256, 1), "fp64", 200, sides="pw"),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def size(v):  # a third each: multiples of 32, even, anything
        r = rng.random()
        return max(16, v // 32 * 32 if r < 1 / 3 else (v // 2 * 2 if r < 2 / 3 else v))

    kind = rng.choice(["steps"] * 8 + ["monitor", "monitor", "loop", "batch", "adjoint"])
    if kind in ("steps", "monitor") and rng.random() < 0.65:
        flow = rng.choice(["bubble", "bubble", "drop", "jet"])
        nx, ny, nz = size(log(24, 256)), size(log(32, 512)), size(log(24, 256))
        precision = rng.choice(["fp32", "fp32", "fp64", "fp16"])
        sides = "jet" if flow == "jet" else rng.choice(["pwp", "pwp", "www", "ppp"])
        nodes = nx * ny * nz * (6 if precision == "fp64" else 1)
        steps = max(1, min(rng.randint(4, 40), int(4e8 / nodes)))
        return _case("", kind, flow, (nx, ny, nz), precision, steps, sides, rng.random() < 0.5)
    if kind in ("steps", "monitor", "loop"):
        flow = rng.choice(["RTI", "drop", "bubble"])
        nx, ny = size(log(32, 512)), size(log(48, 2048))
        precision = rng.choice(["fp64", "fp32", "fp16"])
        steps = rng.randint(5, 20) if kind != "steps" else log(17, 200)
        return _case("", kind, flow, (nx, ny, 1), precision, steps, "pw" if flow == "RTI" else rng.choice(["pw", "ww"]),
                     kind == "steps" and rng.random() < 0.5)
    if kind == "batch":
        return _case("", "batch", "mixed", (256, 512, 1), rng.choice(["fp32", "fp32", "fp64"]), rng.randint(17, 40), "pw",
                     rng.random() < 0.5, log(16, 256))
    return _case("", "adjoint", rng.choice(["drop", "bubble"]), (size(log(32, 320)), size(log(48, 320)), 1), "fp64",
                 rng.randint(20, 200), "pw")


# ---------------------------------------------------------------- the flow of a case
def _flow(case, seed):
    """Numbers of the flow: the interface's place and the fluids, drawn from the seed."""
    r = np.random.RandomState(seed % (1 << 31))
    n = [case["nx"], case["ny"], case["nz"]]
    dim = 3 if n[2] > 1 else 2
    jitter = r.uniform(-1.5, 1.5, 3)
    u = r.uniform(0.0, 1.0, 4)
    d = dict(n=n, dim=dim, flow=case["flow"], W=4.0, mobility=0.02, gravity=GRAVITY, sides=case["sides"])
    if case["flow"] == "RTI":
        L = float(n[0])
        d.update(L=L, Re=2000.0 + 1000.0 * u[0], Pe=1.6 * L, Ca=0.2 + 0.1 * u[1], W=5.0, mu_ratio=1.0,
                 rho_ratio=3.0 + u[2], amplitude=0.05 + 0.02 * u[3], center=[0.0, n[1] / 2 + 0.5 + jitter[1], 0.0])
    elif case["flow"] == "jet":
        R = min(n[0], n[2]) / 4.0
        d.update(L=2 * R, We=15.0 + 10.0 * u[0], Re=200.0 + 100.0 * u[1], mu_ratio=2.0, rho_ratio=4.0, velocity=0.01,
                 R=R, gravity=1e-7, center=[n[0] / 2 + jitter[0], n[1] + 0.5, n[2] / 2 + jitter[2]])
    else:
        m = min(n[:dim])
        R = (m / 8.0 if dim == 3 else m / 5.0) * (0.95 + 0.1 * u[0])
        yc = 0.35 * n[1] if case["flow"] == "bubble" else 0.5 * n[1]
        d.update(L=2 * R, We=6.0 + 4.0 * u[1], Re=(30.0 if dim == 3 else 100.0) + 20.0 * u[2], mu_ratio=10.0 + 90.0 * u[3],
                 rho_ratio=100.0 + 900.0 * u[3], R=R, center=[n[0] / 2 + 0.5 + jitter[0], yc + jitter[1], n[2] / 2 + 0.5 + jitter[2]])
    return d


def _config(d):
    n = d["n"]
    kind = {"RTI": "perturbation", "jet": "sphere"}.get(d["flow"], "sphere" if d["dim"] == 3 else "circle")
    extent = [v + 2 for v in n] if d["dim"] == 3 else [n[0], n[1], 1]
    keys = dict(finalStep=1000, outputInterval=1000, reportInterval=1000, N=extent, referenceLength=d["L"],
                gravity=[0, -d["gravity"], 0], interfaceWidth=d["W"], muRatio=d["mu_ratio"], rhoRatio=d["rho_ratio"],
                Re=d["Re"])
    if d["flow"] == "RTI":
        keys.update(Pe=d["Pe"], Ca=d["Ca"])
    else:
        keys.update(We=d["We"], mobility=d["mobility"])
    geo = ['type = "%s"' % kind, "center = %s" % [float(v) for v in d["center"]], "id = 0"]
    if d["flow"] == "RTI":
        geo += ["amplitude = %.17g" % d["amplitude"], "length = [%.17g, 0, 0]" % d["L"]]
    else:
        geo += ["radius = %.17g" % d["R"]]
    if d["flow"] == "jet":
        keys.update(referenceVelocity=d["velocity"])
        types = ["periodic", "periodic", "free convect", "velocity", "periodic", "periodic"]
    else:
        types = [{"p": "periodic", "w": "wall"}[s] for s in d["sides"] for _ in (0, 1)]
    sides = ["x-", "x+", "y-", "y+", "z-", "z+"][: 2 * d["dim"]]
    blocks = []
    for s, t in zip(sides, types):
        value = "\n    value = [0, %.17g, 0]" % -d["velocity"] if t == "velocity" else ""
        blocks.append('  {\n    side = "%s"\n    type = "%s"%s\n  },' % (s, t.replace(" ", ""), value))
    lines = ["case = " + d["flow"]]
    lines += ["%s = %s" % (k, "%.17g" % v if isinstance(v, float) else v) for k, v in keys.items()]
    lines += ["geometry = [", "  {"] + ["    " + g for g in geo] + ["  }", "]", "boundary = ["] + blocks + ["]", ""]
    return "\n".join(lines)


def _with_config(d, use):
    fd, path = tempfile.mkstemp(suffix=".txt")
    try:
        with os.fdopen(fd, "w") as f:
            f.write(_config(d))
        return use(path)
    finally:
        os.unlink(path)


def _member(case, i):
    """Case i of a batch: sizes of a fixed table (32 to 256 by 64 to 512), drops and bubbles in turn."""
    r = np.random.RandomState(12345 + i)
    nx, ny = 32 * int(r.randint(1, 9)), 64 + 32 * int(r.randint(0, 15))
    return dict(case, flow="bubble" if i % 2 else "drop", nx=nx, ny=ny, nz=1)


# ---------------------------------------------------------------- prepare and run
def prepare(case, seed):
    kind, precision = case["kind"], case["precision"]
    if kind == "batch":
        b = cb.Batch([_config(_flow(_member(case, i), seed * 1009 + i)) for i in range(case["count"])], precision, texts=True)
        b.init()
        if case["tuned"]:
            b.autotune(3)
        views = [b.case(i) for i in range(case["count"])]
        nodes = [v.interior[0] * v.interior[1] for v in views]
        st = dict(batch=b, views=views, at=np.concatenate([[0], np.cumsum(nodes)]),
                  c=torch.zeros(sum(nodes), dtype=torch.float64, device="cuda"),
                  vel=torch.zeros(2 * sum(nodes), dtype=torch.float64, device="cuda"))
        return dict(case=case, **st)
    d = _flow(case, seed)
    if kind == "loop":
        def build(path):
            idata = cb.InputData(path, precision)
            da = cb.DataArray(idata)
            eq = cb.NSAllen(idata, DA=da)
            eq.initialCondition()
            da.updateDevice()
            eq.deviceInitializer()
            return dict(case=case, eq=eq, da=da)
        return _with_config(d, build)
    s = _with_config(d, lambda path: cb.Solver(path, precision))
    if kind == "adjoint":
        target = np.array([d["center"][0] + 5.0, d["center"][1] - 8.0, 0.0])
        return dict(case=case, s=s, target=target)
    stream = torch.cuda.Stream()
    s.set_stream(stream.cuda_stream)
    s.init(on_device=True)
    if case["tuned"]:
        s.autotune(3)
    shape = tuple(v for v in reversed(s.interior[: s.dim]))
    return dict(case=case, s=s, stream=stream, c=torch.zeros(shape, dtype=torch.float64, device="cuda"),
                vel=torch.zeros((s.dim,) + shape, dtype=torch.float64, device="cuda"))


def run(state):
    case = state["case"]
    kind, steps, single = case["kind"], case["steps"], case["precision"] != "fp64"
    if kind == "batch":
        b, at = state["batch"], state["at"]
        b.solve(steps)
        for i, v in enumerate(state["views"]):
            v.field_device("c", state["c"].data_ptr() + 8 * int(at[i]), int(at[i + 1] - at[i]))
            v.field_device("vel", state["vel"].data_ptr() + 16 * int(at[i]), 2 * int(at[i + 1] - at[i]))
        mass, kinetic = b.monitors()
        if not single:
            return dict(c=state["c"], vel=state["vel"], mass=mass, kinetic=kinetic)
        out = dict(c=state["c"].float(), vel=state["vel"].float(), mass=mass.astype(np.float32),
                   kinetic=kinetic.astype(np.float32))
        torch.cuda.current_stream().synchronize()  # the batch's next pass writes the same buffers
        return out
    if kind == "loop":
        for _ in range(steps):
            state["eq"].solve()
        h = state["da"].updateHost()
        return {k: h[k].astype(np.float32) for k in h} if single else dict(h)
    s = state["s"]
    if kind == "adjoint":
        J, g0, gp = s.adjoint(steps, state["target"], checkpoint_every=0)
        return dict(J=J, dc0=g0, dparams=gp)
    out = {}
    if kind == "monitor":
        seen = [s.solve_monitored(1) for _ in range(steps)]
        out["monitors"] = np.array(seen, dtype=np.float32 if single else np.float64)
    else:
        s.solve(steps)
    c, vel = state["c"], state["vel"]
    s.field_device("c", c.data_ptr(), c.numel())
    s.field_device("vel", vel.data_ptr(), vel.numel())
    if single:  # the state is held in 32 bits or less
        with torch.cuda.stream(state["stream"]):
            c, vel = c.float(), vel.float()
    return dict(c=c, vel=vel, **out)


def work(case):
    """Per lattice update: f and g read and written once, c and u read and written once; the
    outputs written once.  Operations: the moment form of the update."""
    dim = 3 if case["nz"] > 1 else 2
    q = 19 if dim == 3 else 9
    pop, aux = {"fp64": (8, 8), "fp32": (4, 4), "fp16": (2, 4)}[case["precision"]]
    per = 4 * q * pop + 2 * (dim + 1) * aux
    nodes = case["nx"] * case["ny"] * case["nz"]
    flops = 620 if dim == 3 else 300
    if case["kind"] == "batch":
        nodes = sum(m["nx"] * m["ny"] for m in (_member(case, i) for i in range(case["count"])))
    out = (dim + 1) * aux * nodes
    passes = 1
    if case["kind"] == "loop":
        out = (dim + 3) * aux * nodes
    if case["kind"] == "adjoint":
        passes, out = 3, 8 * nodes  # forward, and a reverse sweep over stored states and adjoints
    return dict(bytes=float(passes * per * nodes * case["steps"] + out),
                flops=float(passes * flops * nodes * case["steps"]))


# ---------------------------------------------------------------- the same in 64 bits
_E3 = ([0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1, 0, 0, 0, 0],
       [0, 0, 0, 1, -1, 0, 0, 1, -1, -1, 1, 0, 0, 0, 0, 1, -1, 1, -1],
       [0, 0, 0, 0, 0, 1, -1, 0, 0, 0, 0, 1, -1, -1, 1, 1, -1, -1, 1])
_E2 = ([0, 1, 0, -1, 0, 1, -1, -1, 1], [0, 0, 1, 0, -1, 1, 1, -1, -1], [0] * 9)


class _Plain:
    """Two-phase Allen-Cahn lattice Boltzmann step (D2Q9 / D3Q19, weighted MRT) in plain torch
    FP64, one whole-field operation at a time; fields are indexed [z, y, x]."""

    def __init__(self, d):
        self.d, dim = d, d["dim"]
        self.e = _E3 if dim == 3 else _E2
        self.Q = len(self.e[0])
        sq = [sum(abs(self.e[a][q]) for a in range(3)) for q in range(self.Q)]
        self.w = [{0: 1 / 3, 1: 1 / 18, 2: 1 / 36}[v] if dim == 3 else {0: 4 / 9, 1: 1 / 9, 2: 1 / 36}[v] for v in sq]
        self.opp = [next(o for o in range(self.Q) if all(self.e[a][o] == -self.e[a][q] for a in range(3)))
                    for q in range(self.Q)]
        g, L = d["gravity"], d["L"]
        self.rho_h, self.rho_l = 1.0, 1.0 / d["rho_ratio"]
        if d["flow"] == "RTI":
            mu = math.sqrt(g * L) * L / d["Re"]
            sigma, self.M = mu * math.sqrt(g * L) / d["Ca"], math.sqrt(g * L) * L / d["Pe"]
        else:
            sigma, self.M = g * L * L / d["We"], d["mobility"]
            mu = math.sqrt(g * (self.rho_h - self.rho_l) * L ** 3) / d["Re"]
        self.tau_h, self.tau_l = 3.0 * mu, 3.0 * mu / d["mu_ratio"] / self.rho_l
        self.W = d["W"]
        self.kappa, self.beta = 1.5 * sigma * self.W, 8.0 * sigma / self.W
        self.wall = [s == "w" for s in d["sides"]] + [False] * (3 - len(d["sides"]))
        n = d["n"]
        co = [torch.arange(0, n[a] + 2, dtype=torch.float64, device="cuda") for a in range(dim)]
        if dim == 2:
            co.append(torch.zeros(1, dtype=torch.float64, device="cuda"))
        x, y, z = co[0][None, None, :], co[1][None, :, None], co[2][:, None, None]
        c0 = d["center"]
        if d["flow"] == "RTI":
            sd = y - (d["amplitude"] * d["L"] * torch.cos(2 * math.pi * x / d["L"]) + c0[1]) + 0 * z
        else:
            sd = torch.sqrt((x - c0[0]) ** 2 + (y - c0[1]) ** 2 + ((z - c0[2]) ** 2 if dim == 3 else 0 * z)) - d["R"]
        t = torch.tanh(2.0 * sd / self.W)
        ghosted = 0.5 - 0.5 * t if d["flow"] == "drop" else 0.5 + 0.5 * t
        inner = (slice(1, -1) if dim == 3 else slice(None), slice(1, -1), slice(1, -1))
        c = ghosted[inner].clone()
        mu_c, dc = self.stencils(ghosted)
        rho = self.rho_l + c * (self.rho_h - self.rho_l)
        p = {"drop": 1.0, "bubble": -1.0, "RTI": 0.0}[d["flow"]] * c * sigma / (L / 2) / (rho / 3)
        zero = torch.zeros_like(c)
        u = [zero] * dim
        hlp = (1 - 4 * (c - 0.5) ** 2) / self.W
        nrm = self.normal(dc)
        g0 = [c * self.w[q] - 0.5 * self.w[q] * hlp * self.edot(q, nrm) + zero for q in range(self.Q)]
        f0 = [p * self.w[q] for q in range(self.Q)]
        self.c, self.u = c, u
        self.collide(f0, g0, c, mu_c, dc, u, p)

    def edot(self, q, v):
        s = 0.0
        for a in range(len(v)):
            if self.e[a][q]:
                s = s + v[a] if self.e[a][q] > 0 else s - v[a]
        return s

    def normal(self, dc):
        m = torch.sqrt(sum(v * v for v in dc)) + 1e-32
        return [v / m for v in dc]

    def stencils(self, G):
        """mu and grad c from c with its ghost layer."""
        dim, n = self.d["dim"], self.d["n"]

        def at(i, j, k):
            z = slice(1 + k, 1 + k + n[2]) if dim == 3 else slice(None)
            return G[z, 1 + j:1 + j + n[1], 1 + i:1 + i + n[0]]

        ks = (-1, 0, 1) if dim == 3 else (0,)
        c = at(0, 0, 0)
        lap, dc = 0.0, [0.0] * dim
        wl = {1: 20 / 48, 2: 6 / 48, 3: 1 / 48} if dim == 3 else {1: 4 / 6, 2: 1 / 6}
        wg = {1: 2 / 9, 2: 1 / 18, 3: 1 / 72} if dim == 3 else {1: 1 / 3, 2: 1 / 12}
        for i in (-1, 0, 1):
            for j in (-1, 0, 1):
                for k in ks:
                    m = abs(i) + abs(j) + abs(k)
                    if not m:
                        continue
                    v = at(i, j, k)
                    lap = lap + wl[m] * (v - c)
                    for a, s in enumerate((i, j, k)[:dim]):
                        if s:
                            dc[a] = dc[a] + s * wg[m] * v
        return 4 * self.beta * c * (c - 1) * (c - 0.5) - self.kappa * lap, dc

    def equilibrium(self, q, u, u2):
        eu = self.edot(q, u)
        return self.w[q] * (3 * eu + 4.5 * eu * eu - 1.5 * u2)

    def tau(self, c):
        t = self.tau_l + c * (self.tau_h - self.tau_l)
        t = torch.where(c < 0, torch.full_like(c, self.tau_l), t)
        return torch.where(c > 1, torch.full_like(c, self.tau_h), t)

    def moments(self, f, p, u):
        """Second moments of the non-equilibrium part, and their deviators."""
        dim = self.d["dim"]
        S = {}
        for a in range(dim):
            for b in range(a, dim):
                s = 0.0
                for q in range(self.Q):
                    w = self.e[a][q] * self.e[b][q]
                    if w:
                        s = s + w * f[q]
                S[a, b] = s - u[a] * u[b] - (p / 3 if a == b else 0.0)
        tr = sum(S[a, a] for a in range(dim)) / dim
        dev = {k: v - tr if k[0] == k[1] else v for k, v in S.items()}
        return tr, dev

    def force(self, f, c, p, mu, dc, u):
        dim, rho = self.d["dim"], self.rho_l + c * (self.rho_h - self.rho_l)
        drho, tau = self.rho_h - self.rho_l, self.tau(c)
        s = 1 / (tau + 0.5)
        tr, dev = self.moments(f, p, u)
        F = []
        for a in range(dim):
            visc = sum((s * dev[min(a, b), max(a, b)] + (tr if a == b else 0.0)) * dc[b] for b in range(dim))
            F.append(mu * dc[a] - p * drho / 3 * dc[a] - tau * visc * drho)
        weight = {"RTI": rho, "bubble": rho - self.rho_h, "drop": rho - self.rho_l}[self.d["flow"]]
        F[1] = F[1] - weight * self.d["gravity"]
        return F, rho, s, dev

    def collide(self, f, g, c, mu, dc, u, p):
        """Post-collision populations: g relaxes at one rate; of f only the traceless stress
        is relaxed at s, every other moment at 1."""
        dim = self.d["dim"]
        F, rho, s, dev = self.force(f, c, p, mu, dc, u)
        nrm = self.normal(dc)
        pref = 3 * self.M * (1 - 4 * (c - 0.5) ** 2) / self.W
        wc = 1 / (0.5 + 3 * self.M)
        u2 = sum(v * v for v in u)
        self.f, self.g = [], []
        for q in range(self.Q):
            ga = self.equilibrium(q, u, u2)
            self.g.append(g[q] * (1 - wc) + wc * (c * (ga + self.w[q]) + self.w[q] * pref * self.edot(q, nrm)))
            e = [self.e[a][q] for a in range(dim)]
            if dim == 3:
                phi = sum(9.0 * e[a] * e[b] * dev[a, b] for a in range(3) for b in range(a + 1, 3))
                phi = phi + 0.75 * (2 * e[0] ** 2 - e[1] ** 2 - e[2] ** 2) * (2 * dev[0, 0] - dev[1, 1] - dev[2, 2])
                phi = phi + 2.25 * (e[1] ** 2 - e[2] ** 2) * (dev[1, 1] - dev[2, 2])
            else:
                phi = 9.0 * e[0] * e[1] * dev[0, 1] + 2.25 * (e[0] ** 2 - e[1] ** 2) * (dev[0, 0] - dev[1, 1])
            self.f.append(p * self.w[q] + ga + 1.5 * self.w[q] * self.edot(q, F) / rho - (s - 1) * self.w[q] * phi)
        self.u = u

    def stream(self, f):
        """Pull streaming; a source behind a wall gives the node's own opposite population."""
        out = []
        for q in range(self.Q):
            ez, ey, ex = self.e[2][q], self.e[1][q], self.e[0][q]
            v = torch.roll(f[q], (ez, ey, ex), (0, 1, 2)) if q else f[q].clone()
            for axis, e in ((0, ez), (1, ey), (2, ex)):
                if e and self.wall[2 - axis]:
                    layer = [slice(None)] * 3
                    layer[axis] = slice(0, 1) if e > 0 else slice(-1, None)
                    v[tuple(layer)] = f[self.opp[q]][tuple(layer)]
            out.append(v)
        return out

    def step(self):
        dim, n = self.d["dim"], self.d["n"]
        f, g, old = self.stream(self.f), self.stream(self.g), self.c
        c = sum(g)
        # the ghost layer holds the previous step's c: mirrored at walls, wrapped else
        G = old
        for axis in (2, 1, 0) if dim == 3 else (2, 1):
            m = G.shape[axis]
            lo, hi = (0, m - 1) if self.wall[2 - axis] else (m - 1, 0)
            G = torch.cat([G.narrow(axis, lo, 1), G, G.narrow(axis, hi, 1)], axis)
        z = slice(1, 1 + n[2]) if dim == 3 else slice(None)
        G[z, 1:1 + n[1], 1:1 + n[0]] = c
        mu, dc = self.stencils(G)
        p = sum(f)
        F, rho, _, _ = self.force(f, c, p, mu, dc, self.u)
        u = []
        for a in range(dim):
            j = sum(self.e[a][q] * f[q] for q in range(self.Q) if self.e[a][q])
            u.append(j + 0.5 * F[a] / rho)
        self.c, self.p, self.rho = c, p, rho
        self.collide(f, g, c, mu, dc, u, p)


def exact(case, seed):
    nodes = case["nx"] * case["ny"] * case["nz"]
    # the batch and the gradient are many runs; the host loop's arrays hold lagged ghost layers
    if case["kind"] in ("batch", "adjoint", "loop") or case["flow"] == "jet" or nodes * case["steps"] > 8e8:
        return None
    m = _Plain(_flow(case, seed))
    seen = []
    for _ in range(case["steps"]):
        m.step()
        if case["kind"] == "monitor":
            ke = 0.5 * (m.rho_l + m.c * (m.rho_h - m.rho_l)) * sum(v * v for v in m.u)
            seen.append((float(m.c.sum()), float(ke.sum())))
    c, vel = m.c, torch.stack(m.u)
    if m.d["dim"] == 2:
        c, vel = c[0], vel[:, 0]
    out = dict(c=c, vel=vel)
    if case["precision"] == "fp16":
        out["vel"] = None  # half-precision populations leave few digits of the young flow's velocity
    if seen:
        out["monitors"] = np.array(seen) if case["precision"] != "fp16" else None
    return out
