"""Performance cases of the dipolar Gross-Pitaevskii solver.

Every case is a piece of a user's program, called through the package's public
entry points (gpe.Solver, gpe.Batch, gpe.Server):

* "solve": a phase of the step loop (imaginary or real time, FP64 or mixed
  precision) on a kept handle, then mu / E and psi read back, as the drop-in
  programs do between their phases;
* "observe": the observables and density cuts written after a phase;
* "batch": many independent solves stepped together;
* "serve": requests submitted to the request server and waited for.

exact() restates the step in torch at 64 bits: each Crank-Nicolson sweep is the
dense matrix that the line recurrence amounts to, the dipolar convolution a
torch FFT, the integrals Simpson weights.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dbec-gp-mpi-cuda_b200"))
import gpe  # noqa: E402

REF_PI = 3.14159265358979  # the programs' value of pi
SIDES = sorted(n for n in {2 ** a * 3 ** b * 5 ** c for a in range(1, 10) for b in range(6) for c in range(4)} if 16 <= n <= 512)


def _case(name, kind, mode, mixed, grid, dx, trap, g, gd, steps, rms_every=0, ramp=False, count=1):
    return {"name": name, "kind": kind, "mode": mode, "mixed": mixed, "nx": grid[0], "ny": grid[1], "nz": grid[2],
            "dx": dx, "gamma": trap[0], "nu": trap[1], "lambda": trap[2], "g": g, "gd": gd, "steps": steps,
            "rms_every": rms_every, "ramp": ramp, "count": count}


def listed():
    aniso, pancake = (0.5, 1.0, 1.5), (1.0, 1.0, 4.0)
    return [
        # the smallest call: a few steps of a test-sized grid, all latency
        _case("imag_24x20x16", "solve", "imag", False, (24, 20, 16), 0.25, aniso, 50., 10., 4),
        # the small ground state: 64^3, FP64, imaginary time
        _case("imag_64", "solve", "imag", False, (64, 64, 64), 0.25, aniso, 100., 30., 100),
        # the shipped imaginary-time input's grid, with the ramp of the couplings and rms samples of its phases
        _case("imag_128x96x80_ramp", "solve", "imag", False, (128, 96, 80), 0.2, (1., 1., 1.5), 150., 30., 100, 25, True),
        # real time on sides with factors 3 and 5, a rms sample every 10 steps (the dynamics output)
        _case("real_90x100x72", "solve", "real", False, (90, 100, 72), 0.25, aniso, 100., 20., 50, 10),
        # the headline: real time, complex128, 256^3, a rms sample every 100 steps
        _case("real_256", "solve", "real", False, (256, 256, 256), 0.2, pancake, 200., 80., 100, 100),
        # its ground state: imaginary time, FP64, 256^3
        _case("imag_256", "solve", "imag", False, (256, 256, 256), 0.2, pancake, 200., 60., 100),
        # the same in mixed precision
        _case("mixed_imag_256", "solve", "imag", True, (256, 256, 256), 0.2, pancake, 200., 60., 100),
        # the large mixed-precision ground state
        _case("mixed_imag_512x512x256", "solve", "imag", True, (512, 512, 256), 0.25, aniso, 100., 30., 50),
        # mixed precision in real time, a middling grid with factors 3 and 5
        _case("mixed_real_160x144x120", "solve", "real", True, (160, 144, 120), 0.2, pancake, 120., 25., 100, 20),
        # observables and density cuts of a 256^3 real-time state
        _case("observe_real_256", "observe", "real", False, (256, 256, 256), 0.2, pancake, 200., 80., 0),
        # 64 independent mixed-precision ground states, grids 48^3 ... 128^3
        _case("batch_64", "batch", "imag", True, (128, 128, 128), 0.2, aniso, 400., 0.2, 50, count=64),
        # requests to the server: ground states and real-time runs, FP64, grids 48^3 ... 128^3
        _case("serve_12", "serve", "both", False, (128, 128, 128), 0.2, aniso, 400., 0.2, 200, count=12),
    ]


def _sides(rng, top, mixed):
    """A grid of even 5-smooth sides, its volume spread over the logarithm up to `top` points."""
    while True:
        want = math.exp(rng.uniform(math.log(16 ** 3), math.log(top)))
        skew = [math.exp(rng.uniform(-0.35, 0.35)) for _ in range(3)]
        side = [want ** (1 / 3) * s / math.prod(skew) ** (1 / 3) for s in skew]
        grid = [min(SIDES, key=lambda n: abs(math.log(n / s))) for s in side]
        if math.prod(grid) <= top and not (mixed and grid[2] % 4):
            return tuple(grid)


def draw(rng):
    kind = rng.choice(["solve"] * 7 + ["observe", "batch", "serve"])
    mode, mixed = rng.choice(["imag", "real"]), rng.random() < 0.5
    trap = (rng.uniform(0.5, 2.), rng.uniform(0.5, 2.), rng.uniform(0.5, 4.))
    g = rng.uniform(20., 400.)
    gd = rng.uniform(0., 0.2) * g
    dx = rng.uniform(0.15, 0.3)
    if kind == "batch":
        c = _case("", kind, "imag", True, (128, 128, 128), dx, trap, 400., 0.2, rng.randint(10, 50), count=rng.randint(3, 64))
    elif kind == "serve":
        c = _case("", kind, "both", False, (128, 128, 128), dx, trap, 400., 0.2, rng.randint(50, 200), count=rng.randint(1, 12))
    else:
        grid = _sides(rng, 2 ** 25 if mixed else 2 ** 24, mixed)
        steps = 0 if kind == "observe" else max(4, min(rng.randint(4, 100), 2 ** 30 // math.prod(grid)))
        c = _case("", kind, mode, mixed, grid, dx, trap, g, gd, steps, rng.choice([0, 0, 10, 25]) if steps else 0,
                  mode == "imag" and rng.random() < 0.25)
    del c["name"]
    return c


# ------------------------------------------------------------------ inputs
def _one(c, mode=None):
    """Solver parameters of one solve."""
    real = (mode or c["mode"]) == "real"
    dx, n = c["dx"], (c["nx"], c["ny"], c["nz"])
    return dict(real=real, mixed=c["mixed"], n=n, dx=dx, dt=(0.01 if real else 0.1) * dx * dx,
                trap=(c["gamma"], c["nu"], c["lambda"]), cutoff=0.5 * min(n) * dx, g=c["g"], gd=c["gd"])


def _many(c, seed):
    """The solves of a batch or of the server's requests, drawn from the seed; the grids and kinds go round so that
    another seed costs the same.  gd stays below 0.23 g: above it the dipolar attraction may collapse the cloud to
    values that are not finite."""
    rng = random.Random(seed)
    grids = [(48, 48, 48), (64, 64, 64), (96, 96, 64), (128, 128, 128)]
    out = []
    for i in range(c["count"]):
        real = c["kind"] == "serve" and i % 2 == 1
        n = grids[i % 4] if c["kind"] == "batch" else grids[(i // 2) % 4]
        dx = rng.uniform(0.15, 0.3)
        g = rng.uniform(20., c["g"])
        out.append(dict(real=real, mixed=c["mixed"], n=n, dx=dx, dt=(0.01 if real else 0.1) * dx * dx,
                        trap=(rng.uniform(0.5, 2.), rng.uniform(0.5, 2.), rng.uniform(0.5, 8.)),
                        cutoff=0.5 * min(n) * dx, g=g, gd=rng.uniform(0., c["gd"]) * g))
    return out


def _params(q):
    return gpe.make_params(gpe.MODE_REAL if q["real"] else gpe.MODE_IMAG, *q["n"], q["dx"], q["dx"], q["dx"], q["dt"],
                           *q["trap"], q["cutoff"], precision=gpe.PREC_MIXED if q["mixed"] else gpe.PREC_FP64)


def _mesh(q):
    return [(torch.arange(n, dtype=torch.float64, device="cuda") - n // 2) * q["dx"] for n in q["n"]]


def _psi(q, seed):
    """A cloud near the trap's ground state: a Gaussian a little off in place and width, modulated by long waves, with
    a slow phase in real time; normalised."""
    rng = random.Random(seed)
    x, y, z = _mesh(q)
    parts = []
    for r, t in zip((x, y, z), q["trap"]):
        w = t * rng.uniform(0.6, 1.1)
        r = r - rng.uniform(-0.2, 0.2)
        parts.append(torch.exp(-0.5 * w * r * r) * (1. + rng.uniform(0.05, 0.2) * torch.cos(rng.uniform(0.5, 1.5) * r + rng.uniform(0., 6.))))
    psi = parts[0][:, None, None] * parts[1][None, :, None] * parts[2][None, None, :]
    psi = psi / torch.sqrt(torch.sum(psi * psi) * q["dx"] ** 3)
    if q["real"]:
        k = [rng.uniform(-0.3, 0.3) for _ in range(3)]
        psi = psi * torch.exp(1j * (k[0] * x[:, None, None] + k[1] * y[None, :, None] + k[2] * z[None, None, :]))
    return psi


def _host(n, real):
    """A page-locked host array for psi, kept by the program."""
    return torch.empty(n, dtype=torch.complex128 if real else torch.float64, pin_memory=True).numpy()


def _ramp(c):
    return (c["g"] / c["steps"], c["gd"] / c["steps"]) if c["ramp"] and c["steps"] else (0., 0.)


def prepare(case, seed):
    if case["kind"] == "serve":
        return {"case": case, "solves": _many(case, seed), "server": gpe.Server(150 << 30)}
    if case["kind"] == "batch":
        qs = _many(case, seed)
        b = gpe.Batch([_params(q) for q in qs], [q["g"] for q in qs], [q["gd"] for q in qs])
        for i, q in enumerate(qs):
            b.solver(i).set_psi(_psi(q, seed + i).cpu().numpy())
        flat, views, at = _host(sum(math.prod(q["n"]) for q in qs), False), [], 0
        for q in qs:
            views.append(flat[at:at + math.prod(q["n"])].reshape(q["n"]))
            at += math.prod(q["n"])
        return {"case": case, "batch": b, "flat": flat, "views": views}
    q = _one(case)
    s = gpe.Solver(_params(q))
    s.set_psi(_psi(q, seed).cpu().numpy())
    return {"case": case, "q": q, "solver": s, "out": _host(q["n"], q["real"])}


def run(state):
    c = state["case"]
    if c["kind"] == "serve":
        sv = state["server"]
        ids = [sv.submit(_params(q), gpe.REQ_EVOLVE if q["real"] else gpe.REQ_GROUND, q["g"], q["gd"], tol=1e-14,
                         check_every=100, max_steps=c["steps"]) for q in state["solves"]]
        res = [sv.wait(i, 60.) for i in ids]
        return {"status": np.array([r.status for r in res]), "steps": np.array([r.steps for r in res]),
                "mu": np.array([r.mu for r in res]), "en": np.array([r.en for r in res]),
                "norm": np.array([r.norm for r in res]), "rms": np.array([list(r.rms) for r in res])}
    if c["kind"] == "batch":
        state["batch"].run(c["steps"])
        for i, v in enumerate(state["views"]):
            state["batch"].solver(i).get_psi(out=v)
        return {"psi": state["flat"]}
    s, q = state["solver"], state["q"]
    if c["kind"] == "observe":
        norm = s.calcnorm(False)
        mu, en = s.calcmuen(q["g"], q["gd"])
        out = {"norm": norm, "mu": mu, "en": en, "rms": s.calcrms()}
        for k in ("1d_x", "1d_y", "1d_z", "2d_xy", "2d_xz", "2d_yz", "3d_xy0"):
            out["den" + k] = s.density(k)
        return out
    dg, dgd = _ramp(c)
    g0, gd0 = (0., 0.) if c["ramp"] else (q["g"], q["gd"])
    g, gd, norm, rms = s.run(c["steps"], g0, gd0, dg, dgd, rms_every=c["rms_every"])
    mu, en = s.calcmuen(g, gd)
    out = {"mu": mu, "en": en, "psi": s.get_psi(out=state["out"])}
    if not q["real"]:
        out["norm"] = norm
    if rms is not None:
        out["rms"] = rms
    return out


# -------------------------------------------------------------------- work
def _step_work(q):
    """One split step: the convolution's five axis passes and the three sweeps each read and write their array once
    (psi 8 times, the half spectrum 8 times, the kernel once)."""
    n = math.prod(q["n"])
    r = 4 if q["mixed"] else 8
    half = (q["n"][2] // 2 + 1) / q["n"][2]
    cx = 2 if q["real"] else 1
    log = sum(math.log2(m) for m in q["n"])
    return n * (8 * r * cx + 8 * half * 2 * r + half * r), n * (5. * log + 3 * (26 if q["real"] else 8) + 40)


def work(case):
    if case["kind"] in ("batch", "serve"):
        qs = _many(case, 0)
        w = [_step_work(q) for q in qs]
        return {"bytes": case["steps"] * sum(b for b, _ in w), "flops": case["steps"] * sum(f for _, f in w)}
    q = _one(case)
    n, psi = math.prod(q["n"]), (4 if q["mixed"] else 8) * (2 if q["real"] else 1)
    b, f = _step_work(q)
    if case["kind"] == "observe":
        # psi read for the norm, mu / E, rms, the three line integrals of the 1D and 2D outputs; one convolution
        conv = b - n * psi * 6
        return {"bytes": n * psi * 9 + conv, "flops": f + 60. * n}
    obs = -(-case["steps"] // case["rms_every"]) if case["rms_every"] and not q["real"] else 0
    return {"bytes": case["steps"] * b + n * psi * (2 + obs) + b - n * psi * 6 + n * 8 * (2 if q["real"] else 1),
            "flops": case["steps"] * f + 60. * n}


def tolerance(case):
    # against exact(): FP64 4e-15 ... 8e-14, mixed imaginary time 1e-6, mixed real time 4e-6 (the FP32 storage of psi)
    if case["mixed"]:
        return {"rel": 2e-5 if case["mode"] == "real" else 5e-6}
    return {"rel": 1e-11 if case["kind"] == "serve" else 1e-12}


# ------------------------------------------------------------------- exact
def _sweep_matrix(n, q):
    """The dense matrix of one Crank-Nicolson sweep of a line of n points (par = 1)."""
    c = q["dt"] / (q["dx"] * q["dx"]) / 2.
    if q["real"]:
        A0, A0r, A, mA = 1. + 1j * c, 1. - 1j * c, -0.5j * c, 0.5j * c
    else:
        A0, A0r, A, mA = 1. + c, 1. - c, -0.5 * c, 0.5 * c
    t = np.complex128 if q["real"] else np.float64
    al, ga = np.zeros(n - 1, t), np.zeros(n - 1, t)
    ga[n - 2] = -1. / A0
    for i in range(n - 2, 0, -1):
        al[i - 1] = A * ga[i]
        ga[i - 1] = -1. / (A0 + A * al[i - 1])
    p = np.eye(n, dtype=t)
    be = np.zeros((n - 1, n), t)
    be[n - 2] = p[n - 1]
    for i in range(n - 2, 0, -1):
        r = mA * p[i + 1] + A0r * p[i] - A * p[i - 1]
        be[i - 1] = ga[i] * (A * be[i] - r)
    o = np.zeros((n, n), t)
    for i in range(n - 2):
        o[i + 1] = al[i] * o[i] + be[i]
    return torch.from_numpy(o).cuda()


def _simpson(n, h):
    m = n if n % 2 else n - 1
    w = torch.zeros(n, dtype=torch.float64)
    w[1:m - 1:2] = 4.
    w[2:m - 1:2] = 2.
    w[0] = w[m - 1] = 1.
    if n % 2 == 0:
        w[n - 1] += 1.25
        w[n - 2] += 2.
        w[n - 3] -= 0.25
    return w.cuda() * h / 3.


def _fd4(f, axis, h):
    f = f.movedim(axis, 0)
    d = torch.zeros_like(f)
    d[1] = (f[2] - f[0]) / (2. * h)
    d[-2] = (f[-1] - f[-3]) / (2. * h)
    d[2:-2] = (f[:-4] - 8. * f[1:-3] + 8. * f[3:-1] - f[4:]) / (12. * h)
    return d.movedim(0, axis)


class _Exact:
    """The solve in torch at 64 bits."""

    def __init__(self, q, psi):
        self.q, self.psi = q, psi
        n, h = q["n"], q["dx"]
        k2 = []
        for a, m in enumerate(n):
            i = torch.arange(m, dtype=torch.float64, device="cuda") if a < 2 else torch.arange(m // 2 + 1, dtype=torch.float64, device="cuda")
            if a < 2:
                i = torch.minimum(i, m - i)
            k2.append((i * (2. * REF_PI / (m * h))) ** 2)
        s = k2[0][:, None, None] + k2[1][None, :, None] + k2[2][None, None, :]
        kr = torch.sqrt(s) * q["cutoff"]
        self.u = 4. * REF_PI * (3. * k2[2][None, None, :] / s - 1.) / 3. * (1. + 3. * torch.cos(kr) / kr ** 2 - 3. * torch.sin(kr) / kr ** 3)
        self.u[0, 0, 0] = 0.
        x = _mesh(q)
        t = q["trap"]
        self.x2 = [v * v for v in x]
        self.v = 0.5 * (t[0] ** 2 * self.x2[0][:, None, None] + t[1] ** 2 * self.x2[1][None, :, None] + t[2] ** 2 * self.x2[2][None, None, :])
        self.m = [_sweep_matrix(k, q) for k in n]
        self.w = [_simpson(k, h) for k in n]

    def dens(self):
        return self.psi.real ** 2 + self.psi.imag ** 2 if self.q["real"] else self.psi ** 2

    def phi(self, rho):
        p = torch.fft.irfftn(torch.fft.rfftn(rho) * self.u, s=self.q["n"])
        p[-1, :-1, :-1] = p[0, :-1, :-1]
        p[:-1, -1, :-1] = p[:-1, 0, :-1]
        p[:-1, :-1, -1] = p[:-1, :-1, 0]
        return p

    def integral(self, f):
        return torch.einsum("xyz,x,y,z->", f, *self.w).item() if f.numel() < 1 << 20 else \
            (self.w[0] @ ((f @ self.w[2]) @ self.w[1])).item()

    def step(self, g, gd):
        rho = self.dens()
        e = self.v + g * rho
        e += gd * self.phi(rho)
        e *= self.q["dt"]
        self.psi = self.psi * (torch.exp(-1j * e) if self.q["real"] else torch.exp(-e))
        n = self.q["n"]
        self.psi = (self.m[0] @ self.psi.reshape(n[0], -1)).reshape(n)
        self.psi = torch.matmul(self.m[1], self.psi)
        self.psi = self.psi @ self.m[2].T
        if not self.q["real"]:
            nrm = self.norm()
            self.psi = self.psi / nrm
            return nrm

    def norm(self):
        return math.sqrt(self.integral(self.dens()))

    def rms(self):
        rho = self.dens()
        w = self.w
        rz = rho @ w[2]
        m = [torch.dot(w[0] * self.x2[0], rz @ w[1]).item(), torch.dot(w[0], rz @ (w[1] * self.x2[1])).item(),
             torch.dot(w[0], (rho @ (w[2] * self.x2[2])) @ w[1]).item()]
        return [math.sqrt(sum(m))] + [math.sqrt(v) for v in m]

    def muen(self, g, gd):
        a = torch.abs(self.psi) if self.q["real"] else self.psi
        rho = self.dens()
        d = sum(_fd4(a, k, self.q["dx"]) ** 2 for k in range(3)) / 2.
        lin = g * rho + gd * self.phi(rho)
        return self.integral((self.v + lin) * rho + d), self.integral((self.v + 0.5 * lin) * rho + d)


def _gauss(q):
    t = q["trap"]
    x = _mesh(q)
    c = math.sqrt(REF_PI * math.sqrt(REF_PI / (t[0] * t[1] * t[2])))
    e = t[0] * (x[0] ** 2)[:, None, None] + t[1] * (x[1] ** 2)[None, :, None] + t[2] * (x[2] ** 2)[None, None, :]
    p = torch.exp(-0.5 * e) / c
    return p.to(torch.complex128) if q["real"] else p


def exact(case, seed):
    if case["kind"] == "serve":
        out = {"status": None, "steps": None, "mu": [], "en": [], "norm": [], "rms": []}
        for q in _many(case, seed):
            e = _Exact(q, _gauss(q))
            if not q["real"]:
                e.psi = e.psi / e.norm()
            for _ in range(case["steps"]):
                e.step(q["g"], q["gd"])
            mu, en = e.muen(q["g"], q["gd"])
            for k, v in (("mu", mu), ("en", en), ("norm", e.norm()), ("rms", e.rms())):
                out[k].append(v)
        return {k: None if v is None else np.array(v) for k, v in out.items()}
    if case["kind"] == "batch":
        flat = []
        for i, q in enumerate(_many(case, seed)):
            e = _Exact(q, _psi(q, seed + i))
            for _ in range(case["steps"]):
                e.step(q["g"], q["gd"])
            flat.append(e.psi.reshape(-1).cpu().numpy())
        return {"psi": np.concatenate(flat)}
    q = _one(case)
    e = _Exact(q, _psi(q, seed))
    if case["kind"] == "observe":
        mu, en = e.muen(q["g"], q["gd"])
        out = {"norm": e.norm(), "mu": mu, "en": en, "rms": np.array(e.rms())}
        rho, x = e.dens(), [v.cpu().numpy() for v in _mesh(q)]
        for a, k in enumerate("xyz"):
            o = [b for b in range(3) if b != a]
            line = torch.tensordot(torch.tensordot(rho, e.w[o[1]], ([o[1]], [0])), e.w[o[0]], ([o[0]], [0])).cpu().numpy()
            out["den1d_" + k] = np.stack([x[a], line], 1).reshape(-1)
        for a, k in ((2, "xy"), (1, "xz"), (0, "yz")):
            f = torch.tensordot(rho, e.w[a], ([a], [0])).cpu().numpy()
            o = [b for b in range(3) if b != a]
            out["den2d_" + k] = np.stack([*np.meshgrid(x[o[0]], x[o[1]], indexing="ij"), f], 2).reshape(-1)
        f = rho[:, :, q["n"][2] // 2].cpu().numpy()
        out["den3d_xy0"] = np.stack([*np.meshgrid(x[0], x[1], indexing="ij"), f], 2).reshape(-1)
        return out
    dg, dgd = _ramp(case)
    g, gd = (0., 0.) if case["ramp"] else (q["g"], q["gd"])
    nrm, rms = None, []
    for k in range(case["steps"]):
        g += dg
        gd += dgd
        nrm = e.step(g, gd)
        if case["rms_every"] and k % case["rms_every"] == 0:
            rms.append(e.rms())
    mu, en = e.muen(g, gd)
    out = {"mu": mu, "en": en, "psi": e.psi.cpu().numpy()}
    if not q["real"]:
        out["norm"] = nrm
    if rms:
        out["rms"] = np.array(rms)
    return out
