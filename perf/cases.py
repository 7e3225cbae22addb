"""What the performance of this framework is measured on: the work a user has it do, through its
public entry points (``native.Chunk``), over the sizes, solvers and options of its decks.

Three kinds of pass:

run      A run of the program on one chunk (run_deck's loop): generate the state on the device,
         ``steps`` implicit time steps, the last one with the field summary, and the resulting
         energy field read back.  Meshes up to about a million cells run their solves to
         convergence; the large ones over a capped window of iterations, as the benchmark does
         (a whole step there takes thousands of identical iterations).
kernels  A driver that keeps its own CG loop and its fields on the host, and calls the per-kernel
         entry points where the reference calls its kernels.
adjoint  One gradient: a recorded run of time steps and its reverse sweep.

The inputs are random rectangles (and circles) of material on a 10 x 10 domain, as in the decks of
the tests and of the benchmark; the seed decides where they lie and what they are made of.
"""
import math
import random

import numpy as np
import torch

from tealeaf_ref_gb300 import deck as dk
from tealeaf_ref_gb300 import native

DOMAIN = 10.0
DT = 0.004
EPS = 1.0e-15


def _case(name=None, **kw):
    c = dict(kind="run", solver="cg", nx=256, ny=256, steps=1, max_iters=10000, precond="none", coefficient=2,
             reflective=False, halo=1, precision="fp64", inner=10, presteps=20, epslim=1.0, rects=8, circles=0)
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the reference's smallest benchmark deck: ten time steps on 10 x 10 cells, all latency
        _case("cg_10", nx=10, ny=10, steps=10, coefficient=1, rects=4),
        # the small synthetic workload: a whole run of ten time steps on 256 x 256
        _case("cg_256", nx=256, ny=256, steps=10, max_iters=5000, rects=3),
        # a ragged mid-size mesh with the diagonal preconditioner and reflecting walls
        _case("cg_diag_777x1013", nx=777, ny=1013, steps=2, precond="jac_diag", reflective=True, circles=2),
        # the reference's default input deck (PPCG, halo depth 2, 124 inner steps) for one time step
        _case("ppcg_1000", solver="ppcg", nx=1000, ny=1000, coefficient=1, halo=2, inner=124, presteps=25, rects=4),
        # the headline workload: the largest mesh, FP64 CG
        _case("cg_8192", nx=8192, ny=8192, max_iters=200, rects=16, circles=4),
        # the 4096 x 4096 workload with each of the other solvers
        _case("jacobi_4096", solver="jacobi", nx=4096, ny=4096, max_iters=100),
        _case("cheby_4096", solver="chebyshev", nx=4096, ny=4096, max_iters=200, epslim=1e30),
        _case("ppcg_4096", solver="ppcg", nx=4096, ny=4096, max_iters=40, epslim=1e30),
        # the precision form solved to the FP64 form's accuracy: CG, and PPCG's FP32 inner steps
        _case("mixed_cg_2048", nx=2048, ny=2048, precision="mixed", max_iters=50000),
        _case("mixed_ppcg_1999x1500", solver="ppcg", nx=1999, ny=1500, precision="mixed", max_iters=50000),
        # a driver with its own CG loop over the drop-in kernels, odd sizes
        _case("kernels_3001x1999", kind="kernels", nx=3001, ny=1999, max_iters=20, precond="jac_diag"),
        # the gradient of a loss on the final temperature through two time steps
        _case("adjoint_512", kind="adjoint", nx=512, ny=512, steps=2, max_iters=50000),
    ]


def draw(rng):
    def sides(lo, hi):
        side = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        aspect = math.exp(rng.uniform(-0.6, 0.6))
        return tuple(max(lo, min(hi, int(round(x)))) for x in (side * aspect, side / aspect))

    kind = rng.choices(["run", "mixed", "kernels", "adjoint"], [60, 16, 12, 12])[0]
    kw = dict(coefficient=rng.choice([1, 2, 2]), rects=rng.randint(3, 16), circles=rng.choice([0, 0, 2, 4]),
              precond=rng.choices(["none", "jac_diag", "jac_block"], [60, 30, 10])[0])
    if kind == "adjoint":
        nx, ny = sides(32, 700)
        return _case(**dict(kw, kind="adjoint", nx=nx, ny=ny, steps=rng.randint(1, 3), max_iters=50000, precond="none"))
    if kind == "kernels":
        nx, ny = sides(16, 6000)
        return _case(**dict(kw, kind="kernels", nx=nx, ny=ny, max_iters=rng.randint(5, 40)))
    if kind == "mixed":
        nx, ny = sides(200, 2200)
        if kw["precond"] == "jac_block":
            kw["precond"] = "none"
        return _case(**dict(kw, precision="mixed", solver=rng.choice(["cg", "cg", "ppcg", "chebyshev"]), nx=nx, ny=ny,
                            max_iters=50000))
    kw["solver"] = rng.choices(["cg", "ppcg", "chebyshev", "jacobi"], [50, 20, 15, 15])[0]
    nx, ny = sides(8, 8192)
    small = nx * ny <= 1200 * 1200
    if kw["solver"] == "cg":
        kw["reflective"] = rng.random() < 0.25
    if kw["solver"] == "jacobi":
        kw.update(max_iters=rng.randint(50, 200) if small else rng.randint(30, 100), precond="none")
    elif kw["solver"] == "chebyshev":
        kw.update(max_iters=rng.randint(60, 500) if small else rng.randint(40, 160), epslim=1e30)
    elif kw["solver"] == "ppcg":
        kw.update(inner=rng.choice([5, 10, 10, 20]), halo=1 if kw["precond"] == "jac_block" else rng.choice([1, 1, 2]))
        if not small:
            kw.update(max_iters=rng.randint(30, 36), epslim=1e30, inner=rng.choice([5, 10]))
    else:
        kw.update(max_iters=10000 if small else rng.randint(40, 200))
    kw["steps"] = rng.randint(1, 4) if small else 1
    return _case(**dict(kw, nx=nx, ny=ny))


# ---- the inputs ---------------------------------------------------------------------------------
def _states(case, seed):
    """Rectangles and circles of material on the ambient state (density, energy, geometry, extents)."""
    rng = random.Random(int(seed) * 7919 + 13)
    out = [dict(density=100.0, energy=1.0e-4, geometry=1, xmin=0.0, xmax=0.0, ymin=0.0, ymax=0.0, radius=0.0)]
    for _ in range(case["rects"]):
        w, h = rng.uniform(0.5, 3.0), rng.uniform(0.5, 3.0)
        x, y = rng.uniform(0.0, DOMAIN - w), rng.uniform(0.0, DOMAIN - h)
        out.append(dict(density=rng.uniform(0.1, 1.0), energy=rng.uniform(1.0, 25.0), geometry=1, xmin=x, xmax=x + w,
                        ymin=y, ymax=y + h, radius=0.0))
    for _ in range(case["circles"]):
        r = rng.uniform(0.2, 1.0)
        out.append(dict(density=0.1, energy=25.0, geometry=2, xmin=rng.uniform(r, DOMAIN - r), xmax=0.0,
                        ymin=rng.uniform(r, DOMAIN - r), ymax=0.0, radius=r))
    return out


def _deck(case, seed):
    return dk.Deck(states=[dk.State(**s) for s in _states(case, seed)], x_cells=case["nx"], y_cells=case["ny"],
                   xmin=0.0, ymin=0.0, xmax=DOMAIN, ymax=DOMAIN, initial_timestep=DT, max_iters=case["max_iters"],
                   eps=EPS, solver=case["solver"], coefficient=case["coefficient"], preconditioner=case["precond"],
                   reflective_boundary=case["reflective"], halo_depth=case["halo"], ch_cg_presteps=case["presteps"],
                   ch_cg_epslim=case["epslim"], ppcg_inner_steps=case["inner"], end_step=case["steps"])


def _u_bar(case, seed):
    g = np.random.default_rng(int(seed) + 77)
    return g.uniform(-1.0, 1.0, (case["ny"], case["nx"]))


def prepare(case, seed):
    deck = _deck(case, seed)
    chunk = native.Chunk.from_deck(deck, generate=False)
    state = dict(kind=case["kind"], deck=deck, chunk=chunk, steps=case["steps"],
                 opts=native.opts_from_deck(deck, case["precision"]))
    shape = (case["ny"], case["nx"])
    if case["kind"] == "adjoint":
        state["u_bar"] = _u_bar(case, seed)
        return state
    state["pinned"] = native.PinnedArray(shape)
    if case["kind"] == "kernels":
        chunk.generate(deck)
        hosts = [native.PinnedArray(shape) for _ in range(2)]
        for name, h in zip(("density", "energy1"), hosts):
            chunk.download(name, h.array)
        state.update(density=hosts[0], energy=hosts[1], iters=case["max_iters"])
    return state


# ---- the passes ---------------------------------------------------------------------------------
def run(state):
    chunk = state["chunk"]
    if state["kind"] == "kernels":
        return _run_kernels(state)
    chunk.generate(state["deck"])
    if state["kind"] == "adjoint":
        chunk.adjoint_begin(state["steps"])
        for _ in range(state["steps"]):
            chunk.record_step(state["opts"], DT)
        density_bar, energy_bar, _ = chunk.adjoint_backward(state["u_bar"])
        return {"density_bar": density_bar, "energy_bar": energy_bar}
    chunk.reset_eigen()
    for _ in range(state["steps"] - 1):
        chunk.tea_leaf(state["opts"], DT)
    _, summary = chunk.tea_leaf_summary(state["opts"], DT)
    return {"energy": chunk.download("energy1", state["pinned"].array), "summary": summary}


def _run_kernels(state):
    chunk = state["chunk"]
    chunk.upload_state(state["density"].array, state["energy"].array)
    chunk.common_init(DT)
    chunk.calc_residual()
    chunk.calc_2norm(1)
    rro = chunk.cg_init()
    for _ in range(state["iters"]):
        pw = chunk.cg_calc_w()
        rrn = chunk.cg_calc_ur(rro / pw)
        chunk.cg_calc_p(rrn / rro)
        rro = rrn
    chunk.finalise()
    return {"energy": chunk.download("energy1", state["pinned"].array), "rro": rro}


def _typical_iterations(case):
    """Iterations of one time step: the cap of a window, or what a converged solve of this size takes."""
    cells = case["nx"] * case["ny"]
    if case["kind"] == "run" and (case["solver"] == "jacobi" or case["max_iters"] < 1000):
        return case["max_iters"]
    n = max(5, int(1.1 * math.sqrt(cells) if case["coefficient"] == 1 else 2.2 * math.sqrt(cells)))
    return min(n, case["max_iters"])


def work(case):
    # bytes and operations of one iteration: FP64 CG 96 B (12 streams) and 10, Jacobi 40 B and 15,
    # Chebyshev 56 B and 8, PPCG inner 64 B and 8; the precision form half the bytes
    cells = case["nx"] * case["ny"]
    n = _typical_iterations(case) * case["steps"]
    if case["kind"] == "adjoint":
        n *= 2
    per = {"cg": (96, 20), "jacobi": (40, 15), "chebyshev": (56, 16), "ppcg": (96, 20)}[case["solver"]]
    b, f = per[0] * n, per[1] * n
    if case["solver"] == "ppcg" and case["max_iters"] < 1000:
        b, f = b + 64 * case["inner"] * (n - case["presteps"]), f + 16 * case["inner"] * (n - case["presteps"])
    if case["precision"] == "mixed":
        b //= 2
    if case["precond"] != "none":
        b, f = b + 16 * n, f + 2 * n
    return {"bytes": cells * b, "flops": cells * f}


# ---- the same in plain torch --------------------------------------------------------------------
class _Plain:
    """The chunk's state, operator and solves in 64 bits, from the equations."""

    def __init__(self, case, seed):
        self.case = case
        self.dev = dev = "cuda" if torch.cuda.is_available() else "cpu"
        nx, ny = case["nx"], case["ny"]
        self.dx, self.dy = DOMAIN / nx, DOMAIN / ny
        self.rx, self.ry = DT / self.dx ** 2, DT / self.dy ** 2
        f64 = dict(dtype=torch.float64, device=dev)
        x0, y0 = torch.arange(nx, **f64) * self.dx, torch.arange(ny, **f64) * self.dy
        x1, y1 = torch.arange(1, nx + 1, **f64) * self.dx, torch.arange(1, ny + 1, **f64) * self.dy
        self.rho = torch.empty(ny, nx, **f64)
        self.e = torch.empty(ny, nx, **f64)
        for i, s in enumerate(_states(case, seed)):
            if i == 0:
                self.rho.fill_(s["density"])
                self.e.fill_(s["energy"])
                continue
            ax, ay = self.dx / 100.0, self.dy / 100.0  # the extents are drawn in by a hundredth of a cell
            if s["geometry"] == 1:
                mx = (x1 >= s["xmin"] + ax) & (x0 < s["xmax"] - ax)
                my = (y1 >= s["ymin"] + ay) & (y0 < s["ymax"] - ay)
                hit = my[:, None] & mx[None, :]
            else:
                ex, ey = 0.5 * (x0 + x1) - (s["xmin"] + ax), 0.5 * (y0 + y1) - (s["ymin"] + ay)
                hit = torch.sqrt(ex[None, :] ** 2 + ey[:, None] ** 2) <= s["radius"]
            self.rho[hit] = s["density"]
            self.e[hit] = s["energy"]
            del hit
        self.faces()

    def faces(self):
        """Face coefficients between interior cells: rx Kx (ny, nx-1) and ry Ky (ny-1, nx)."""
        w = 1.0 / self.rho if self.case["coefficient"] == 2 else self.rho
        self.w = w
        self.cx = self.rx * (w[:, :-1] + w[:, 1:]) / (2.0 * w[:, :-1] * w[:, 1:])
        self.cy = self.ry * (w[:-1] + w[1:]) / (2.0 * w[:-1] * w[1:])
        self.di = torch.ones_like(w)
        self.di[:, :-1] += self.cx
        self.di[:, 1:] += self.cx
        self.di[:-1] += self.cy
        self.di[1:] += self.cy
        if self.case["reflective"]:  # the walls' faces count in the diagonal preconditioner
            self.wall = torch.zeros_like(w)
            self.wall[:, 0] += self.rx / w[:, 0]
            self.wall[:, -1] += self.rx / w[:, -1]
            self.wall[0] += self.ry / w[0]
            self.wall[-1] += self.ry / w[-1]
        else:
            self.wall = 0.0

    def A(self, v):
        o = v * self.di
        o[:, :-1] -= self.cx * v[:, 1:]
        o[:, 1:] -= self.cx * v[:, :-1]
        o[:-1] -= self.cy * v[1:]
        o[1:] -= self.cy * v[:-1]
        return o

    def cg(self, u, b, max_iters, stop=None):
        """CG from u: (u, r, alphas, betas, converged); stop(n, error): leave before iteration n."""
        mi = 1.0 / (self.di + self.wall) if self.case["precond"] == "jac_diag" else None
        r = b - self.A(u)
        goal = EPS * math.sqrt(float((r * r).sum()))
        z = r if mi is None else mi * r
        p = z.clone()
        rro = float((r * z).sum())
        err = math.sqrt(float((r * r).sum()))
        al, be, n = [], [], 1
        # a window's cap ends the reference's loop; a converged solve goes on until the residual
        # has fallen as far as it does in 64 bits
        while n <= max_iters:
            if stop and stop(n, err):
                return u, r, al, be, False
            w = self.A(p)
            a = rro / float((p * w).sum())
            u = u.add_(p, alpha=a)
            r.add_(w, alpha=-a)
            z = r if mi is None else mi * r
            rrn = float((r * z).sum())
            al.append(a)
            be.append(rrn / rro)
            p.mul_(rrn / rro).add_(z)
            rro = rrn
            err = math.sqrt(abs(rrn))
            if err < goal:
                return u, r, al, be, True
            n += 1
        return u, r, al, be, True

    def spectrum(self, al, be):
        n = len(al)
        d = np.array([1.0 / al[i] + (be[i - 1] / al[i - 1] if i else 0.0) for i in range(n)])
        off = np.array([math.sqrt(be[i]) / al[i] for i in range(n - 1)])
        ev = np.linalg.eigvalsh(np.diag(d) + np.diag(off, 1) + np.diag(off, -1))
        return ev[0] * 0.95, ev[-1] * 1.05

    @staticmethod
    def coefficients(lo, hi, n):
        theta, delta = (hi + lo) / 2.0, (hi - lo) / 2.0
        sigma = theta / delta
        rho, a, b = 1.0 / sigma, [0.0], [0.0]
        for _ in range(n):
            new = 1.0 / (2.0 * sigma - rho)
            a.append(new * rho)
            b.append(2.0 * new / delta)
            rho = new
        return theta, a, b

    def solve(self, b):
        """One time step's u from u = b, as the case's solver leaves it."""
        c = self.case
        window = c["max_iters"] if c["max_iters"] < 1000 else None
        u = b.clone()
        if c["solver"] == "jacobi":
            for _ in range(c["max_iters"]):
                s = b.clone()
                s[:, :-1] += self.cx * u[:, 1:]
                s[:, 1:] += self.cx * u[:, :-1]
                s[:-1] += self.cy * u[1:]
                s[1:] += self.cy * u[:-1]
                u = s / self.di
            return u
        if c["solver"] == "cg" or window is None:
            return self.cg(u, b, window or 60000)[0]
        u, r, al, be, done = self.cg(u, b, window, lambda n, err: n >= c["presteps"] and err <= c["epslim"])
        if done:
            return u
        n = len(al) + 1
        lo, hi = self.spectrum(al, be)
        mi = 1.0 / self.di if c["precond"] == "jac_diag" else None
        pre = (lambda v: v) if mi is None else (lambda v: mi * v)
        theta, a, bb = self.coefficients(lo, hi, max(window + 2, c["inner"]))
        if c["solver"] == "chebyshev":
            p = pre(b - self.A(u)) / theta
            u = u + p
            for i in range(1, window - n + 2):
                p = a[i] * p + bb[i] * pre(b - self.A(u))
                u = u + p
            return u

        def inner(r):
            sd = pre(r) / theta
            rt, ut = r.clone(), sd.clone()
            for i in range(1, c["inner"] + 1):
                rt = rt - self.A(sd)
                sd = a[i] * sd + bb[i] * pre(rt)
                ut = ut + sd
            return ut

        z = inner(r)
        p = z.clone()
        for _ in range(n, window + 1):
            w = self.A(p)
            rro = float((z * r).sum())
            alpha = rro / float((p * w).sum())
            old = r.clone()
            u = u + alpha * p
            r = r - alpha * w
            z = inner(r)
            p = z + (float(((r - old) * z).sum()) / rro) * p
        return u


def exact(case, seed):
    cells, window = case["nx"] * case["ny"], case["max_iters"] < 1000
    if case["precond"] == "jac_block" and (window or case["kind"] == "kernels"):
        return None
    if window and case["solver"] != "cg" and (case["reflective"] or cells > 8e6 * 3):
        return None
    c = dict(case, precond="none") if not window and case["precond"] == "jac_block" else case
    m = _Plain(c, seed)
    vol = m.dx * m.dy
    if case["kind"] == "kernels":
        b = m.e * m.rho
        u, r, al, be, _ = m.cg(b.clone(), b, case["max_iters"])
        mi = 1.0 / m.di if case["precond"] == "jac_diag" else 1.0
        return {"energy": (u / m.rho).cpu().numpy(), "rro": float((r * r * mi).sum())}
    if case["kind"] == "adjoint":
        return _exact_adjoint(m, torch.from_numpy(_u_bar(case, seed)).to(m.dev))
    e = m.e
    for _ in range(case["steps"]):
        u = m.solve(e * m.rho)
        e = u / m.rho
    mass = vol * m.rho
    summary = np.array([vol * cells, float(mass.sum()), float((mass * e).sum()), float((mass * u).sum())])
    return {"energy": e.cpu().numpy(), "summary": summary}


def _exact_adjoint(m, u_bar):
    es, us, e = [], [], m.e
    for _ in range(m.case["steps"]):
        es.append(e)
        us.append(m.cg(e * m.rho, e * m.rho, 60000)[0])
        e = us[-1] / m.rho
    rho_bar, e_bar = torch.zeros_like(m.rho), torch.zeros_like(m.rho)
    for i, (e, u) in reversed(list(enumerate(zip(es, us)))):
        rhs = e_bar / m.rho + (u_bar if i == len(es) - 1 else 0.0)
        rho_bar -= e_bar * u / m.rho ** 2
        lam = m.cg(rhs.clone(), rhs, 60000)[0]
        rho_bar += lam * e
        # K = (wl + wr) / (2 wl wr): dK/dw = -1 / (2 w^2) on either side; w = rho or 1 / rho
        kx = -m.rx * (lam[:, 1:] - lam[:, :-1]) * (u[:, 1:] - u[:, :-1])
        ky = -m.ry * (lam[1:] - lam[:-1]) * (u[1:] - u[:-1])
        k = torch.zeros_like(rho_bar)
        k[:, 1:] += kx
        k[:, :-1] += kx
        k[1:] += ky
        k[:-1] += ky
        rho_bar += 0.5 * k if m.case["coefficient"] == 2 else -k / (2.0 * m.rho ** 2)
        e_bar = lam * m.rho
    return {"density_bar": rho_bar.cpu().numpy(), "energy_bar": e_bar.cpu().numpy()}
