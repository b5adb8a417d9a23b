"""The calls that a user of this framework makes, as measurable cases.

Three public paths, at the sizes of the repository's own decks, tests and
benchmark and at odd sizes between them:

  deck     a whole tea.in run: set-up, timesteps, summaries, the temperature
           field read back (lib.run_deck, per call as the Fortran driver
           calls the C ABI, or device-resident);
  batch    many independent problems of uneven size: fields in, timesteps,
           fields, summaries and iteration counts out (lib.Batch);
  adjoint  the time-stepped loss and its gradient in log-density through the
           torch.autograd.Function (adjoint.time_stepped_loss).

The library keeps one chunk, one batch and one adjoint object per process,
so a deck's state is its text (a run sets up its chunk as a user's run
does), and a batch or an adjoint object of the case's sizes is the plan that
a program keeps while its fields change.
"""
import math
import random

import numpy as np
import torch

from tealeaf_opencl_gb300 import adjoint, decks, lib

DEFAULTS = dict(kind="deck", solver="cg", prec="none", steps=1, eps=1e-15, max_iters=1000,
                halo=1, mode="resident", form="fused", inner=0, presteps=25, after=0,
                mixed=False, inverse=False)


def _case(name, **kw):
    return dict(DEFAULTS, name=name, **kw)


def listed():
    return [
        # the smallest test problem: 10 x 10 Jacobi, one host round trip per sweep
        _case("jacobi_10", solver="jacobi", x=10, y=10, steps=10, mode="per_call"),
        # a small ragged grid through the Fortran driver's own call sequence
        _case("cg_61x47_per_call", x=61, y=47, steps=10, eps=1e-12, mode="per_call"),
        # the benchmark's small CG configuration (diagonal Jacobi to 1e-15)
        _case("cg_512_diag", prec="jac_diag", x=512, y=512, steps=3, max_iters=5000),
        # the 960^2 CG test problem, scalars returned to the host every call
        _case("cg_960_per_call", x=960, y=960, steps=1, max_iters=10000, mode="per_call"),
        # an ordinary odd-sized device-resident CG with the block preconditioner
        _case("cg_1501x1203_block", prec="jac_block", x=1501, y=1203, max_iters=1200,
              form="chain"),
        # the largest CG: every field far larger than L2
        _case("cg_4096_diag", prec="jac_diag", x=4096, y=4096, max_iters=800, form="chain"),
        # the 500^2 PPCG test problem (88 inner steps, halo depth 4)
        _case("ppcg_500", solver="ppcg", x=500, y=500, steps=1, eps=1e-12, max_iters=10000,
              halo=4),
        # the benchmark's headline: PPCG, block Jacobi, 10 inner steps, 4096^2
        _case("ppcg_4096_block", solver="ppcg", prec="jac_block", x=4096, y=4096, steps=2,
              halo=2, form="chain", inner=10, presteps=20, after=60),
        # Chebyshev with the diagonal preconditioner on an odd mid-sized grid
        _case("cheby_1111x901_diag", solver="chebyshev", prec="jac_diag", x=1111, y=901,
              max_iters=1500, eps=1e-10, presteps=20),
        # FP32 inner CG inside FP64 defect correction to a 1e-10 residual
        _case("mixed_2048_diag", prec="jac_diag", x=2048, y=2048, eps=1e-10, max_iters=10000,
              mixed=True),
        # uneven independent problems solved together
        dict(name="batch_40", kind="batch", n=40, lo=64, hi=640, layout=1, steps=2, eps=1e-12,
             max_iters=5000),
        # loss and gradient of a time-stepped solve
        dict(name="adjoint_512", kind="adjoint", x=512, y=512, steps=4, every=2, eps=1e-10,
             max_iters=5000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["deck"] * 6 + ["batch", "adjoint"])
    if kind == "batch":
        lo = _log(rng, 16, 128)
        return dict(kind="batch", n=_log(rng, 4, 64), lo=lo, hi=_log(rng, lo + 1, 640),
                    layout=rng.randrange(1000), steps=rng.choice([1, 2]), eps=1e-12,
                    max_iters=5000)
    if kind == "adjoint":
        steps = rng.choice([2, 3, 4])
        return dict(kind="adjoint", x=_log(rng, 16, 700), y=_log(rng, 16, 700), steps=steps,
                    every=rng.randint(1, steps), eps=1e-10, max_iters=5000)
    solver = rng.choice(["jacobi", "cg", "cg", "cg", "ppcg", "chebyshev"])
    prec = "none" if solver == "jacobi" else rng.choice(["none", "jac_diag", "jac_block"])
    side = _log(rng, 8, 1024 if solver == "jacobi" else 4000)
    c = dict(DEFAULTS, solver=solver, prec=prec, x=side, y=max(4, int(side * rng.uniform(0.6, 1.0))),
             mode=rng.choice(["resident", "per_call"]), form=rng.choice(["fused", "chain"]),
             halo=rng.choice([1, 1, 2, 3]), steps=rng.choice([1, 2]),
             inverse=rng.random() < 0.15, eps=rng.choice([1e-15, 1e-12, 1e-10]))
    cells = c["x"] * c["y"]
    c["max_iters"] = int(min(2000, 8e9 / cells / c["steps"]))
    if solver == "ppcg":
        c["inner"] = rng.choice([4, 10, 25])
        c["presteps"] = rng.randint(15, 30)
        c["after"] = max(2, int(min(60, 1.2e10 / cells / c["steps"] / (c["inner"] + 1))))
    if solver == "cg" and prec == "jac_diag" and side > 100 and rng.random() < 0.3:
        c.update(mixed=True, eps=1e-10, steps=1, inverse=False, max_iters=2000)
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _states(seed):
    """The five-state layout of the repository's decks with each density and
    energy within 10 % of its value."""
    r = random.Random(1000003 * int(seed) + 17)
    t = decks.FIVE_STATE_TABLE
    return dict(t, density=[v * r.uniform(0.9, 1.1) for v in t["density"]],
                energy=[v * r.uniform(0.9, 1.1) for v in t["energy"]])


def _deck(case, seed):
    s = _states(seed)
    lines = ["*tea", "state 1 density=%r energy=%r" % (s["density"][0], s["energy"][0])]
    for k in range(1, 5):
        lines.append("state %d density=%r energy=%r geometry=rectangle xmin=%r xmax=%r ymin=%r "
                     "ymax=%r" % (k + 1, s["density"][k], s["energy"][k], s["xmin"][k],
                                  s["xmax"][k], s["ymin"][k], s["ymax"][k]))
    lines += ["x_cells=%d" % case["x"], "y_cells=%d" % case["y"], "xmin=0.0", "ymin=0.0",
              "xmax=10.0", "ymax=10.0", "initial_timestep=0.004",
              "end_step=%d" % case["steps"], "summary_frequency=10",
              "tl_max_iters=%d" % case["max_iters"], "tl_use_%s" % case["solver"],
              "tl_eps=%r" % case["eps"], "halo_depth=%d" % case["halo"],
              "tl_ch_cg_presteps=%d" % case["presteps"], "tl_arithmetic %s" % case["form"]]
    if case["prec"] != "none":
        lines.append("tl_preconditioner_type=%s" % case["prec"])
    if case["inner"]:
        lines.append("tl_ppcg_inner_steps=%d" % case["inner"])
    if case["mixed"]:
        lines += ["tl_mixed_precision", "tl_mixed_inner_eps=1e-5"]
    if case["inverse"]:
        lines.append("tl_coefficient_inverse_density")
    return "\n".join(lines + ["*endtea"]) + "\n"


def _batch_problems(case, seed):
    layout = random.Random(case["layout"])
    r = random.Random(1000003 * int(seed) + 29)
    out = []
    for _ in range(case["n"]):
        p = dict(x=layout.randint(case["lo"], case["hi"]), y=layout.randint(case["lo"], case["hi"]),
                 states=[])
        for _ in range(layout.randint(2, 6)):
            x0, x1 = sorted(layout.uniform(0.0, 10.0) for _ in range(2))
            y0, y1 = sorted(layout.uniform(0.0, 10.0) for _ in range(2))
            dens = math.exp(layout.uniform(math.log(0.05), math.log(200.0)))
            p["states"].append(dict(density=dens * r.uniform(0.9, 1.1),
                                    energy=layout.uniform(1e-4, 25.0) * r.uniform(0.9, 1.1),
                                    xmin=x0, xmax=x1, ymin=y0, ymax=y1))
        out.append(p)
    return out


def _adjoint_fields(case, seed):
    """(log density, energy, u_obs): smooth random fields on the GPU."""
    g = torch.Generator().manual_seed(int(seed) + 7)
    shape = (case["y"], case["x"])

    def smooth(scale):
        coarse = torch.randn((1, 1, 6, 6), generator=g, dtype=torch.float64)
        f = torch.nn.functional.interpolate(coarse, size=shape, mode="bicubic",
                                            align_corners=True)[0, 0]
        return scale * f.cuda()

    log_density = math.log(5.0) + smooth(0.7)
    energy = torch.exp(smooth(0.8))
    u_obs = torch.exp(log_density) * energy * torch.exp(smooth(0.1))
    return log_density.contiguous(), energy.contiguous(), u_obs.contiguous()


_kept = {}  # the process's batch and adjoint object: what a program keeps


def _plan(kind, key, make):
    if _kept.get(kind, (None,))[0] != key:
        lib.load().tea_gb300_set_arithmetic(lib.ARITHMETIC["fused"])
        _kept.pop(kind, None)
        _kept[kind] = (key, make())
    return _kept[kind][1]


def _batch_plan(state):
    return _plan("batch", state["sizes"], lambda: lib.Batch(list(state["sizes"]), prec="jac_diag"))


def _adjoint_plan(state):
    return _plan("adjoint", state["shape"], lambda: lib.Adjoint(state["shape"][1], state["shape"][0]))


def prepare(case, seed):
    if case["kind"] == "deck":
        lib.load()
        return dict(case=case, deck=_deck(case, seed))
    if case["kind"] == "batch":
        problems = _batch_problems(case, seed)
        state = dict(case=case, sizes=tuple((p["x"], p["y"]) for p in problems),
                     fields=[decks.paint(p) for p in problems])
        _batch_plan(state)
        return state
    fields = _adjoint_fields(case, seed)
    state = dict(case=case, shape=(case["y"], case["x"]), fields=fields,
                 cfg=lib.Adjoint.config(case["steps"], 0.004, case["eps"], case["max_iters"],
                                        case["every"]))
    _adjoint_plan(state)
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "deck":
        mode = lib.DRIVER_RESIDENT if case["mode"] == "resident" else lib.DRIVER_PER_CALL
        infos = lib.run_deck(state["deck"], mode=mode, cap_after_switch=case["after"])
        last = infos[-1]
        return dict(u=lib.read_field("u"),
                    summary=np.array([last.vol, last.mass, last.ie, last.temp]),
                    iterations=np.array([[i.iterations, i.inner_iterations, i.outer_corrections,
                                          i.switch_iteration] for i in infos]))
    if case["kind"] == "batch":
        b = _batch_plan(state)
        for i, (density, energy) in enumerate(state["fields"]):
            b.set_fields(i, density, energy)
        b.run(case["steps"], 0.004, case["eps"], case["max_iters"])
        n = case["n"]
        return dict(u=np.concatenate([b.read(i, "u").reshape(-1) for i in range(n)]),
                    summary=np.array([b.summary(i) for i in range(n)]),
                    iterations=np.array([b.iterations(i) for i in range(n)]))
    log_density, energy, u_obs = state["fields"]
    theta = log_density.detach().requires_grad_(True)
    loss = adjoint.time_stepped_loss(theta, energy, u_obs, _adjoint_plan(state), state["cfg"])
    loss.backward()
    return dict(loss=loss.detach(), grad=theta.grad)


def work(case):
    """Nominal: fields in and out once and, as flops, one operator
    application and its vector updates (about 24 per cell and iteration),
    for the iterations that the five-state problem takes at this size."""
    if case["kind"] == "batch":
        sizes = [(p["x"], p["y"]) for p in _batch_problems(case, 0)]
        cells = sum(x * y for x, y in sizes)
        iters = sum(x * y * min(case["max_iters"], 0.7 * max(x, y)) for x, y in sizes)
        return {"bytes": 24.0 * cells, "flops": 24.0 * iters * case["steps"]}
    cells = case["x"] * case["y"]
    side = max(case["x"], case["y"])
    if case["kind"] == "adjoint":
        solves = 3 * case["steps"] - min(case["every"], case["steps"])
        return {"bytes": 40.0 * cells, "flops": 24.0 * cells * 0.4 * side * solves}
    if case["solver"] == "jacobi":
        its = min(case["max_iters"], 25 + 10 * side) * case["steps"]
    elif case["solver"] == "ppcg" and case["after"]:
        its = max(case["presteps"], 0.09 * side) + case["steps"] * case["after"] * (case["inner"] + 1)
    elif case["solver"] == "chebyshev":
        its = min(case["max_iters"], 4.0 * side + 25) * case["steps"]
    else:
        its = min(case["max_iters"], 0.9 * side + 10) * case["steps"]
        if case["mixed"]:
            its = 0.6 * side + 10
    return {"bytes": 32.0 * cells, "flops": 24.0 * cells * its}


# ---------------------------------------------------------------------------
# the same results in plain 64-bit torch
# ---------------------------------------------------------------------------

class _Grid:
    """(I + dt L_K) on one chunk with zeroed boundary faces, and M^-1."""

    def __init__(self, density, prec="none", inverse=False, dt=0.004):
        self.y, self.x = density.shape
        dx, dy = 10.0 / float(np.float32(self.x)), 10.0 / float(np.float32(self.y))
        w = 1.0 / density if inverse else density
        self.rx, self.ry = dt / (dx * dx), dt / (dy * dy)
        pad = torch.nn.functional.pad
        kx = (w[:, :-1] + w[:, 1:]) / (2.0 * w[:, :-1] * w[:, 1:]) * self.rx
        ky = (w[:-1] + w[1:]) / (2.0 * w[:-1] * w[1:]) * self.ry
        self.kw, self.ke = pad(kx, (1, 0)), pad(kx, (0, 1))
        self.ks, self.kn = pad(ky, (0, 0, 1, 0)), pad(ky, (0, 0, 0, 1))
        self.diag = 1.0 + (self.kn + self.ks) + (self.ke + self.kw)
        self.prec = prec
        if prec == "jac_block":
            self._block()

    def _block(self):
        """Factors of the tridiagonal blocks of 4 rows of one column."""
        self.cp, self.bfp = torch.zeros_like(self.diag), torch.zeros_like(self.diag)
        for j in range(4):
            a = -self.ks[j::4]
            n = a.shape[0]
            b = self.diag[j::4] if j == 0 else self.diag[j::4] - a * self.cp[j - 1::4][:n]
            self.bfp[j::4] = 1.0 / b
            self.cp[j::4] = -self.kn[j::4] / b

    def a(self, u):
        out = self.diag * u
        out[:, :-1] -= self.ke[:, :-1] * u[:, 1:]
        out[:, 1:] -= self.kw[:, 1:] * u[:, :-1]
        out[:-1] -= self.kn[:-1] * u[1:]
        out[1:] -= self.ks[1:] * u[:-1]
        return out

    def m(self, r):
        if self.prec == "none":
            return r
        if self.prec == "jac_diag":
            return r / self.diag
        z = torch.empty_like(r)
        for j in range(4):
            v = r[j::4]
            if j:
                v = v + self.ks[j::4] * z[j - 1::4][: v.shape[0]]
            z[j::4] = v * self.bfp[j::4]
        for j in (2, 1, 0):
            up = z[j + 1::4]
            n = up.shape[0]
            z[j::4][:n] -= self.cp[j::4][:n] * up
        return z


def _dot(a, b):
    return float((a * b).sum())


def _cg(g, u0, u, eps, max_iters, target=None):
    """Preconditioned CG as the driver runs it."""
    r = u0 - g.a(u)
    target = eps * math.sqrt(_dot(r, r)) if target is None else target
    p = g.m(r).clone()
    rro = _dot(r, p)
    for _ in range(max_iters):
        w = g.a(p)
        alpha = rro / _dot(p, w)
        u = u + alpha * p
        r -= alpha * w
        z = g.m(r)
        rrn = _dot(r, z)
        p = z + (rrn / rro) * p
        rro = rrn
        if math.sqrt(abs(rrn)) < target:
            break
    return u


def _coefficients(lo, hi, n):
    return decks.chebyshev_coefficients(lo, hi, n)


def _eig_range(al, be):
    n = len(al)
    t = np.diag([1.0 / al[i] + (be[i - 1] / al[i - 1] if i else 0.0) for i in range(n)])
    for i in range(n - 1):
        t[i, i + 1] = t[i + 1, i] = math.sqrt(be[i]) / al[i]
    e = np.linalg.eigvalsh(t)
    return e[0] * 0.95, e[-1] * 1.05


def _step(case, g, u, eig):
    """One timestep's solve from u0 = u; returns (u, eigenvalue range)."""
    u0 = u.clone()
    solver, eps, most = case["solver"], case["eps"], case["max_iters"]
    if solver == "jacobi":
        r = u0 - g.a(u)
        target = eps * math.sqrt(_dot(r, r))
        for _ in range(most):
            new = (u0 + g.diag * u - g.a(u)) / g.diag
            err = float((new - u).abs().sum())
            u = new
            if math.sqrt(err) < target:
                break
        return u, eig
    if solver == "cg":
        if case["mixed"]:
            r = u0 - g.a(u)
            return _cg(g, u0, u, 0.0, 20000, 1e-14 * math.sqrt(_dot(r, r))), eig
        return _cg(g, u0, u, eps, most), eig
    inner = case["inner"] or 4 * int(math.sqrt(math.sqrt(case["x"] * case["y"])))
    r = u0 - g.a(u)
    old = initial = math.sqrt(_dot(r, r))
    p = g.m(r).clone()
    rro = _dot(r, p)
    al, be = [], []
    steps, error, estimate, n, switched = 0, 0.0, 0, 1, False
    first, loop_max = eig is None, most
    while n <= loop_max:
        switched = switched or steps > 0 or (not first and solver == "ppcg" and n > 1) or \
            (old <= 1.0 and n >= case["presteps"])
        if switched and steps == 0:
            eig = eig or _eig_range(al, be)
            first = False
            if case["after"]:
                loop_max = min(loop_max, n - 1 + case["after"])
            ca, cb, theta = _coefficients(eig[0], eig[1], inner if solver == "ppcg" else most - n + 2)
        if switched and solver == "chebyshev":
            if steps == 0:
                bb = _dot(u0, u0)
                p = g.m(u0 - g.a(u)) / theta
                u = u + p
            r = u0 - g.a(u)
            p = ca[max(steps, 1) - 1] * p + cb[max(steps, 1) - 1] * g.m(r)
            u = u + p
            if steps == 0:
                old = _dot(r, r)
                s = math.sqrt(eig[1] / eig[0])
                q = math.log(eps * bb / (4.0 * old)) / (2.0 * math.log((s - 1.0) / (s + 1.0)))
                estimate, steps = round(q), 1
            elif n >= estimate and n % 10 == 0:
                error = _dot(r, r)
            steps += 1
        else:
            w = g.a(p)
            alpha = rro / _dot(p, w)
            u = u + alpha * p
            r = r - alpha * w
            z = g.m(r)
            if switched:
                sd = z / theta
                for k in range(inner):
                    u = u + sd
                    r = r - g.a(sd)
                    sd = ca[k] * sd + cb[k] * g.m(r)
                steps += 1
                if g.prec == "none":
                    z = r
            rrn = _dot(r, z)
            if not switched:
                al.append(alpha)
                be.append(rrn / rro)
            p = z + (rrn / rro) * p
            error = rro = rrn
        error = math.sqrt(abs(error))
        if error < eps * initial:
            break
        old = error
        n += 1
    return u, eig


def _paint(case, seed):
    """(density, energy) of the deck: a cell takes the last state whose
    rectangle, shrunk by a hundredth of a cell, meets it."""
    s, x, y = _states(seed), case["x"], case["y"]
    dx, dy = 10.0 / float(np.float32(x)), 10.0 / float(np.float32(y))
    d = torch.full((y, x), s["density"][0], dtype=torch.float64)
    e = torch.full((y, x), s["energy"][0], dtype=torch.float64)
    vx, vy = np.arange(x + 1) * dx, np.arange(y + 1) * dy
    for k in range(1, 5):
        mx = (vx[1:] >= s["xmin"][k] + dx / 100) & (vx[:-1] < s["xmax"][k] - dx / 100)
        my = (vy[1:] >= s["ymin"][k] + dy / 100) & (vy[:-1] < s["ymax"][k] - dy / 100)
        m = torch.from_numpy(my)[:, None] & torch.from_numpy(mx)[None, :]
        d[m], e[m] = s["density"][k], s["energy"][k]
    return d, e


def _summary(density, energy, u):
    y, x = density.shape
    vol = (10.0 / float(np.float32(x))) * (10.0 / float(np.float32(y)))
    return [vol * x * y, float(vol * density.sum()), float((vol * density * energy).sum()),
            float((vol * density * u).sum())]


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def exact(case, seed):
    if case["kind"] == "deck":
        density, energy = (t.to(_device()) for t in _paint(case, seed))
        g, eig = _Grid(density, case["prec"], case["inverse"]), None
        for _ in range(case["steps"]):
            u, eig = _step(case, g, energy * density, eig)
            energy = u / density
        return dict(u=u.cpu().numpy(), summary=np.array(_summary(density, energy, u)),
                    iterations=None)
    if case["kind"] == "batch":
        us, sums = [], []
        for p in _batch_problems(case, seed):
            density, energy = (torch.from_numpy(f).to(_device()) for f in decks.paint(p))
            g = _Grid(density, "jac_diag")
            for _ in range(case["steps"]):
                u0 = energy * density
                u = _cg(g, u0, u0, case["eps"], case["max_iters"])
                energy = u / density
            us.append(u.cpu().numpy().reshape(-1))
            sums.append(_summary(density, energy, u))
        return dict(u=np.concatenate(us), summary=np.array(sums), iterations=None)
    log_density, energy, u_obs = _adjoint_fields(case, seed)
    rho = torch.exp(log_density)
    g = _Grid(rho, "jac_diag")

    def solve(b):
        r = b - g.a(b)
        return _cg(g, b, b, 0.0, 20000, 1e-13 * math.sqrt(_dot(r, r)))

    us = [rho * energy]
    for _ in range(case["steps"]):
        us.append(solve(us[-1]))
    lam = us[-1] - u_obs
    loss = 0.5 * (lam * lam).sum()
    grad = torch.zeros_like(rho)
    for n in range(case["steps"] - 1, -1, -1):
        mu, u = solve(lam), us[n + 1]
        gx, gy = torch.zeros_like(rho), torch.zeros_like(rho)
        fx = -(mu[:, :-1] - mu[:, 1:]) * (u[:, :-1] - u[:, 1:])
        fy = -(mu[:-1] - mu[1:]) * (u[:-1] - u[1:])
        gx[:, :-1] += fx
        gx[:, 1:] += fx
        gy[:-1] += fy
        gy[1:] += fy
        grad += -g.rx / (2.0 * rho) * gx - g.ry / (2.0 * rho) * gy
        lam = mu
    return dict(loss=loss, grad=grad + lam * us[0])
