"""Performance cases of the GB300 Sayram-2D path: what a user of the library has it do, through
its public entry points (capi.Solver, capi.Batch, capi.Server, sayram_step_noalloc).

A pass starts from given states (initial values a program sets or copies in), advances them by a
few backward-Euler steps and reads the result back, so that every pass on the same inputs gives
the same answer. The grids, time steps, step counts and coefficient distributions are those of the
configurations, tests and benchmark of this repository.

  form "solver"   one capi.Solver, as the reference's main loop drives its Solver: set_f, then
                  update() after update() (with the Dirichlet values uploaded anew before each
                  where "bc_each_step" is set, as host/Solver.h does), then f()
  form "run"      one capi.Solver stepped between two saves of a run: set_f, step(n), f()
  form "host"     one capi.Batch of uneven instances, step_host(n) on pinned host buffers
  form "noalloc"  sayram_step_noalloc on the caller's device arrays
  form "server"   capi.Server: requests of different grids and step counts submitted while
                  others run, ticked until all are done, every result polled
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import __graft_entry__

__graft_entry__.load_package()
from sayram2d_gb300 import capi, cases  # noqa: E402

PRECISIONS = {"fp64": 0, "fp32_refine": 1, "fp32_refine_dw": 2}
PRECONDS = {"jacobi": 0, "alpha_line": 1}


def _one(name, form, nx, ny, steps, precision, dt, **kw):
    return {"name": name, "form": form, "nx": nx, "ny": ny, "steps": steps, "precision": precision, "dt": dt,
            "equation": "synthetic", "precond": "alpha_line", **kw}


def _batch(name, n, distinct, lo, hi, steps, precision, dt=1e-2, precond="alpha_line"):
    return {"name": name, "form": "host", "instances": n, "distinct": distinct, "mix": 2024, "lo": lo, "hi": hi,
            "steps": steps, "precision": precision, "dt": dt, "precond": precond}


def listed():
    return [
        # the smallest grids a service sees, stepped one update() at a time: launches and
        # synchronisation are most of it; an odd width, so every row ends in padding
        _one("solver-33x32-fp64", "solver", 33, 32, 20, "fp64", 1e-2),
        # the plain run configuration (configs/c0.ini): 90 x 90, dt = 1e-3 day, FP64
        _one("solver-90x90-fp64", "solver", 90, 90, 20, "fp64", 1e-3),
        # the reference's own run file (80 x 80, D from a table, dt = 2e-3 day) through the drop-in's
        # per-step protocol with the Dirichlet values re-read every step, in the fastest mode
        _one("table-80x80-dw", "solver", 80, 80, 20, "fp32_refine_dw", 2e-3, bc_each_step=True,
             equation="Albert_Young"),
        # one large instance between two saves, the plain FP64 drop-in (1024 x 1024, dt = 1e-2 day)
        _one("run-1024x1024-fp64", "run", 1024, 1024, 4, "fp64", 1e-2),
        # the same instance in the fastest mode
        _one("run-1024x1024-dw", "run", 1024, 1024, 8, "fp32_refine_dw", 1e-2),
        # an odd, elongated grid of the loss-cone case (zero flux on both alpha0 sides)
        _one("run-389x517-lc-dw", "run", 389, 517, 8, "fp32_refine_dw", 2e-3, equation="Albert_Young_LC"),
        # a few uneven instances: too little work to fill the GPU
        _batch("host-24-uneven-dw", 24, 24, 64, 256, 6, "fp32_refine_dw"),
        # the benchmark's batch of uneven instances (nalpha, nE uniform in [64, 256]), cut to a
        # quarter of its instances so that inputs can be made quickly
        _batch("host-1024-uneven-dw", 1024, 64, 64, 256, 4, "fp32_refine_dw"),
        # the batched plain FP64 path on the same distribution
        _batch("host-192-uneven-fp64", 192, 48, 64, 256, 4, "fp64"),
        # FP32 Krylov with IEEE FP64 refinement, and Jacobi scaling alone: the options beside the
        # default ones
        _batch("host-192-uneven-mixed-jacobi", 192, 48, 64, 256, 4, "fp32_refine", precond="jacobi"),
        # the step for callers that may not allocate, on the largest square grid it takes
        _one("noalloc-256x256-fp64", "noalloc", 256, 256, 4, "fp64", 1e-2),
        # continuous batching: requests with n log-uniform in [32, 512], step counts log-uniform,
        # arriving while others are on the GPU
        {"name": "server-48-dw", "form": "server", "requests": 48, "per_tick": 2, "mix": 2024, "lo": 32, "hi": 512,
         "steps_lo": 10, "steps_hi": 80, "precision": "fp32_refine_dw", "dt": 1e-2, "lanes": 2},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: any grid, step count and option the listed forms take."""
    form = rng.choice(["solver", "solver", "run", "run", "host", "host", "noalloc", "server"])
    prec = rng.choice(["fp64", "fp32_refine_dw", "fp32_refine_dw", "fp32_refine"])
    precond = rng.choice(["alpha_line", "alpha_line", "alpha_line", "jacobi"])
    dt = rng.choice([1e-3, 2e-3, 1e-2])
    equation = rng.choice(["synthetic", "synthetic", "Albert_Young", "Albert_Young_LC"])
    if form == "solver":
        return {"form": form, "nx": _log_int(rng, 20, 260), "ny": _log_int(rng, 20, 260), "steps": rng.randint(2, 24),
                "precision": prec, "dt": dt, "equation": equation, "precond": precond,
                "bc_each_step": rng.random() < 0.5}
    if form == "run":
        return {"form": form, "nx": _log_int(rng, 120, 1024), "ny": _log_int(rng, 120, 1024), "steps": rng.randint(2, 4),
                "precision": prec, "dt": dt, "equation": equation, "precond": precond}
    if form == "host":
        n = _log_int(rng, 2, 192)
        lo = rng.randint(24, 96)
        return {"form": form, "instances": n, "distinct": min(n, 32), "mix": rng.randint(0, 9999), "lo": lo,
                "hi": rng.randint(lo + 8, 256), "steps": rng.randint(1, 4), "precision": prec, "dt": dt, "precond": precond}
    if form == "noalloc":
        return {"form": form, "nx": _log_int(rng, 24, 256), "ny": _log_int(rng, 24, 256), "steps": rng.randint(1, 6),
                "precision": "fp64", "dt": dt, "equation": "synthetic", "precond": "alpha_line"}
    return {"form": form, "requests": rng.randint(6, 40), "per_tick": rng.randint(1, 8), "mix": rng.randint(0, 9999),
            "lo": 32, "hi": rng.randint(96, 400), "steps_lo": 5, "steps_hi": rng.randint(20, 60),
            "precision": rng.choice(["fp32_refine_dw", "fp32_refine_dw", "fp64"]), "dt": 1e-2, "lanes": rng.choice([1, 2])}


# ------------------------------------------------------------------------------ inputs
def _table(seed):
    return cases.synthetic_dtable(seed, n_alpha=91, n_E=49)


def _problem(case, seed):
    """(problem, D table or None) of a single-instance case."""
    nx, ny, dt = case["nx"], case["ny"], case["dt"]
    if case["equation"] == "synthetic":
        return cases.synthetic_problem(nx, ny, dt, seed=seed, tau=1.0), None
    mk = cases.albert_young_problem if case["equation"] == "Albert_Young" else cases.albert_young_lc_problem
    zero = np.zeros((nx, ny))
    return mk(nx, ny, dt, D=(zero, zero, zero)), _table(seed)


def _batch_problems(case, seed):
    """(distinct problems, index of the problem of each instance). The sizes are the case's own."""
    n, m = case["instances"], case["distinct"]
    sizes = cases.batch_sizes(m, case["mix"], case["lo"], case["hi"])
    return [cases.batch_instance(k, seed, case["dt"], sizes[k]) for k in range(m)], [k % m for k in range(n)]


def _requests(case, seed):
    """(problem, steps) of each request, in the order they arrive. Grids and step counts are the
    case's own."""
    rng = np.random.default_rng([case["mix"], 5])
    out = []
    for k in range(case["requests"]):
        n = int(round(math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"])))))
        steps = int(round(math.exp(rng.uniform(math.log(case["steps_lo"]), math.log(case["steps_hi"])))))
        out.append((cases.batch_instance(k, seed, case["dt"], (n, n)), steps))
    return out


def _options(case):
    return {"precision": PRECISIONS[case["precision"]], "precond": PRECONDS[case.get("precond", "alpha_line")]}


def prepare(case, seed):
    form = case["form"]
    if form in ("solver", "run"):
        prob, table = _problem(case, seed)
        s = capi.Solver(prob, **_options(case))
        if table is not None:
            s.set_dtable(table)
        return {"case": case, "solver": s, "prob": prob}
    if form == "host":
        distinct, which = _batch_problems(case, seed)
        b = capi.Batch([distinct[k] for k in which], **_options(case))
        n = int(b.offsets[-1])
        f_in = torch.empty(n, dtype=torch.float64, pin_memory=True)
        np.concatenate([distinct[k].f0.ravel() for k in which], out=f_in.numpy())
        return {"case": case, "batch": b, "in": f_in, "out": torch.zeros(n, dtype=torch.float64, pin_memory=True)}
    if form == "noalloc":
        prob, _ = _problem(case, seed)
        dev = lambda a: torch.tensor(np.ascontiguousarray(a, dtype=np.float64), device="cuda")
        keep = {k: dev(getattr(prob, k)) for k in ("x_edges", "y_edges", "G", "Dxx", "Dxy", "Dyy", "inv_tau", "f0")}
        p = capi.sayram_problem()
        p.nx, p.ny, p.dt = prob.nx, prob.ny, prob.dt
        for k in ("x_edges", "y_edges", "G", "Dxx", "Dxy", "Dyy", "inv_tau"):
            setattr(p, k, ctypes.cast(keep[k].data_ptr(), capi._dp))
        p.f0 = capi._dp()
        for side in range(4):
            p.bc[side] = prob.bc[side]
            p.dirichlet[side] = capi._dp()
            if prob.dirichlet[side] is not None:
                keep["dir%d" % side] = dev(prob.dirichlet[side])
                p.dirichlet[side] = ctypes.cast(keep["dir%d" % side].data_ptr(), capi._dp)
        return {"case": case, "p": p, "keep": keep, "out": torch.empty_like(keep["f0"]), "stats": capi.sayram_stats()}
    reqs = _requests(case, seed)
    srv = capi.Server(4e9, max_slots=64, max_side=512, lanes=case["lanes"], split_side=128,
                      precision=PRECISIONS[case["precision"]])
    return {"case": case, "server": srv, "reqs": reqs}


# ------------------------------------------------------------------------------ one pass
def run(state):
    case = state["case"]
    form = case["form"]
    if form in ("solver", "run"):
        s, prob = state["solver"], state["prob"]
        s.set_f(prob.f0)
        if form == "run":
            s.step(case["steps"])
            return s.f()
        for _ in range(case["steps"]):
            if case.get("bc_each_step"):
                for side in range(4):
                    if prob.dirichlet[side] is not None:
                        s.set_dirichlet(side, prob.dirichlet[side])
            s.update()
        return s.f()
    if form == "host":
        state["batch"].step_host(case["steps"], state["in"].data_ptr(), state["out"].data_ptr())
        return state["out"]
    if form == "noalloc":
        rc = capi.load().sayram_step_noalloc(
            ctypes.byref(state["p"]), None, case["steps"], state["keep"]["f0"].data_ptr(), state["out"].data_ptr(),
            torch.cuda.current_stream().cuda_stream, ctypes.byref(state["stats"]))
        capi.check(rc, "sayram_step_noalloc")
        return state["out"]
    srv, reqs = state["server"], state["reqs"]
    ids, sent, done = [], 0, 0
    while done < len(reqs):
        for _ in range(case["per_tick"]):
            if sent < len(reqs):
                ids.append(srv.submit(*reqs[sent]))
                sent += 1
        done += srv.tick()
    return np.concatenate([srv.poll(r)[0].ravel() for r in ids])


# ------------------------------------------------------------------------------ what it takes
def work(case):
    """Bytes: what a step cannot do without -- per cell the state in and out and the coefficients
    that define the system (G, three D's, 1/tau) read once, 8 bytes each -- and for a pass its
    input and output states once more. Operations: 2 per multiply-add of one assembly (~100 per
    cell) and of one preconditioned Krylov iteration with its residual (~50 per cell), the least
    any solve of a changed system takes."""
    def of(cells, steps):
        return cells * (steps * 56.0 + 16.0), cells * steps * 300.0

    if case["form"] == "host":
        mean = 0.5 * (case["lo"] + case["hi"])
        b, f = of(case["instances"] * mean * mean, case["steps"])
    elif case["form"] == "server":
        lo, hi, a, z = case["lo"], case["hi"], case["steps_lo"], case["steps_hi"]
        cells = (hi * hi - lo * lo) / (2.0 * math.log(hi / lo))  # mean of n^2, n log-uniform
        b, f = of(case["requests"] * cells, (z - a) / math.log(z / a))
    else:
        b, f = of(float(case["nx"]) * case["ny"], case["steps"])
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------------------ 64-bit answers
EPS = 2.220446049250313e-16


class _Exact:
    """The same scheme (Gao-Wu two-point fluxes with cross diffusion, backward Euler) on a set of
    instances padded to one size, in plain 64-bit torch: arrays are (instance, row, column) with
    the row along log E; cells outside an instance hold zeros and a unit diagonal."""

    def __init__(self, probs, fields):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        B = len(probs)
        self.NX, self.NY = max(p.nx for p in probs), max(p.ny for p in probs)
        NX, NY = self.NX, self.NY
        self.shapes = [(p.nx, p.ny) for p in probs]
        pad = lambda shape: np.zeros((B,) + shape)
        xe, ye = pad((NX + 1,)), pad((NY + 1,))
        G, Dxx, Dxy, Dyy, it, f = (pad((NY, NX)) for _ in range(6))
        dirv = [pad((NY + 1,)), pad((NY + 1,)), pad((NX + 1,)), pad((NX + 1,))]
        isdir = np.zeros((4, B), dtype=bool)
        for k, p in enumerate(probs):
            nx, ny = p.nx, p.ny
            xe[k, :nx + 1], ye[k, :ny + 1] = p.x_edges, p.y_edges
            xe[k, nx + 1:] = p.x_edges[-1] + 1.0 + np.arange(NX - nx)
            ye[k, ny + 1:] = p.y_edges[-1] + 1.0 + np.arange(NY - ny)
            for dst, src in zip((G, Dxx, Dxy, Dyy, it, f), (p.G, *fields[k], p.inv_tau, p.f0)):
                dst[k, :ny, :nx] = np.asarray(src).T
            for s in range(4):
                if p.bc[s] == 0:
                    isdir[s, k] = True
                    dirv[s][k, :len(p.dirichlet[s])] = p.dirichlet[s]
        t = lambda a: torch.tensor(a, device=self.dev)
        self.nx, self.ny = (t(np.array([s[q] for s in self.shapes])).view(B, 1, 1) for q in (0, 1))
        i, j = torch.arange(NX + 1, device=self.dev).view(1, 1, -1), torch.arange(NY + 1, device=self.dev).view(1, -1, 1)
        self.i, self.j = i, j
        self.inside = (i[..., :-1] < self.nx) & (j[:, :-1] < self.ny)
        xe, ye = t(xe), t(ye)
        dx, dy = (xe[:, 1:] - xe[:, :-1]).unsqueeze(1), (ye[:, 1:] - ye[:, :-1]).unsqueeze(2)
        xc, yc = 0.5 * (xe[:, 1:] + xe[:, :-1]), 0.5 * (ye[:, 1:] + ye[:, :-1])
        wx, wy = torch.zeros_like(xe), torch.zeros_like(ye)  # weight of the lower cell at each vertex line
        wx[:, 1:-1] = (xc[:, 1:] - xe[:, 1:-1]) / (xc[:, 1:] - xc[:, :-1])
        wy[:, 1:-1] = (yc[:, 1:] - ye[:, 1:-1]) / (yc[:, 1:] - yc[:, :-1])
        self.wx, self.wy = wx.unsqueeze(1), wy.unsqueeze(2)
        G = t(G)
        self.a, self.b, self.c = t(Dxx) * G * dy / dx, t(Dyy) * G * dx / dy, t(Dxy) * G
        dt = t(np.array([float(p.dt) for p in probs])).view(B, 1, 1)
        self.ukk = G * dx * dy / dt
        self.diag0 = self.ukk * (1.0 + dt * t(it))
        self.diag0[~self.inside] = 1.0
        self.dirv = [t(dirv[0]).unsqueeze(2), t(dirv[1]).unsqueeze(2), t(dirv[2]).unsqueeze(1), t(dirv[3]).unsqueeze(1)]
        self.isdir = t(isdir).view(4, B, 1, 1)
        self.f = t(f)

    @staticmethod
    def _sh(a, dim, by):
        """a moved by one place along a dimension (zero filled): by = 1 takes each entry's lower
        neighbour, by = -1 its upper one."""
        out = torch.zeros_like(a)
        n = a.shape[dim]
        out.narrow(dim, 1 if by > 0 else 0, n - 1).copy_(a.narrow(dim, 0 if by > 0 else 1, n - 1))
        return out

    def _vertices(self):
        f, i, j, nx, ny = self.f, self.i, self.j, self.nx, self.ny
        B = f.shape[0]
        lo = torch.zeros(B, self.NY, self.NX + 1, dtype=f.dtype, device=self.dev)
        hi = lo.clone()
        lo[..., 1:], hi[..., :-1] = f, f
        row = torch.where(i == 0, hi, torch.where(i >= nx, lo, self.wx * lo + (1.0 - self.wx) * hi))
        dn = torch.zeros(B, self.NY + 1, self.NX + 1, dtype=f.dtype, device=self.dev)
        up = dn.clone()
        dn[:, 1:], up[:, :-1] = row, row
        v = torch.where(j == 0, up, torch.where(j >= ny, dn, self.wy * dn + (1.0 - self.wy) * up))
        on = (i == 0, i == nx, j == 0, j == ny)
        for s in range(4):
            v = torch.where(on[s] & self.isdir[s], self.dirv[s], v)
        return v

    @staticmethod
    def _pair(aK, SK, fK, aL, SL, fL):
        den = aK.abs() + aL.abs() + 2 * EPS
        muK = (aL.abs() + EPS) / den
        muL = 1.0 - muK
        Bn = muL * aL - muK * aK
        return muK * SK + Bn.clamp(min=0) / (fK + EPS), muL * SL + (-Bn).clamp(min=0) / (fL + EPS)

    def assemble(self):
        """Outflow coefficients of every cell to its west, east, south and north neighbours, the
        diagonal and the right-hand side."""
        v, f, sh = self._vertices(), self.f, self._sh
        sw, se, nw, ne = v[:, :-1, :-1], v[:, :-1, 1:], v[:, 1:, :-1], v[:, 1:, 1:]
        one = lambda s, c, p, q: (s - c) * p + (s + c) * q
        aw, ae = one(self.a, self.c, nw, sw), one(self.a, self.c, se, ne)
        as_, an = one(self.b, -self.c, sw, se), one(self.b, -self.c, ne, nw)
        Sx, Sy = 2 * self.a, 2 * self.b
        i, j = self.i[..., :-1], self.j[:, :-1]
        W, eL = self._pair(aw, Sx, f, sh(ae, 2, 1), sh(Sx, 2, 1), sh(f, 2, 1))
        S, nL = self._pair(as_, Sy, f, sh(an, 1, 1), sh(Sy, 1, 1), sh(f, 1, 1))
        zero = torch.zeros_like(f)
        inx, iny = self.inside & (i > 0), self.inside & (j > 0)
        W, eL, S, nL = (torch.where(m, q, zero) for m, q in ((inx, W), (inx, eL), (iny, S), (iny, nL)))
        E, N = sh(eL, 2, -1), sh(nL, 1, -1)
        D, R = self.diag0 + W + E + S + N, self.ukk * f
        edge = (i == 0, i == self.nx - 1, j == 0, j == self.ny - 1)
        for s, (a, S0) in enumerate(((aw, Sx), (ae, Sx), (as_, Sy), (an, Sy))):
            m = edge[s] & self.isdir[s] & self.inside
            D = D + torch.where(m, S0 + (-a).clamp(min=0) / (f + EPS), zero)
            R = R + torch.where(m, a.clamp(min=0), zero)
        return W, E, S, N, D, R

    def step(self):
        W, E, S, N, D, R = self.assemble()
        sh = self._sh
        w, e, s, n = (q / D for q in (E, W, N, S))  # what a row's west, ... neighbour sends into it
        w, e, s, n = sh(w, 2, 1), sh(e, 2, -1), sh(s, 1, 1), sh(n, 1, -1)

        def mul(y):
            t = y.clone()
            t[:, :, 1:].addcmul_(w[:, :, 1:], y[:, :, :-1], value=-1)
            t[:, :, :-1].addcmul_(e[:, :, :-1], y[:, :, 1:], value=-1)
            t[:, 1:].addcmul_(s[:, 1:], y[:, :-1], value=-1)
            t[:, :-1].addcmul_(n[:, :-1], y[:, 1:], value=-1)
            return t

        dot = lambda a, b: (a * b).sum((1, 2), keepdim=True)
        safe = lambda a, b: torch.where(b != 0, a / torch.where(b != 0, b, torch.ones_like(b)), torch.zeros_like(a))
        y, bb = D * self.f, dot(R, R)
        for _ in range(4):  # BiCGSTAB from the true residual each time
            r = R - mul(y)
            if bool((dot(r, r) <= 1e-30 * bb).all()):
                break
            rh, p, rho, goal = r.clone(), r.clone(), dot(r, r), torch.maximum(1e-31 * bb, 1e-20 * dot(r, r))
            for _ in range(400):
                vv = mul(p)
                al = safe(rho, dot(rh, vv))
                q = r - al * vv
                tt = mul(q)
                om = safe(dot(tt, q), dot(tt, tt))
                y = y + al * p + om * q
                r = q - om * tt
                if bool((dot(r, r) <= goal).all()):
                    break
                rho2 = dot(rh, r)
                p = r + safe(rho2, rho) * safe(al, om) * (p - om * vv)
                rho = rho2
        self.f = (y / D) * self.inside

    def get(self, k):
        nx, ny = self.shapes[k]
        return self.f[k, :ny, :nx].T.contiguous().cpu().numpy()


def _table_fields(prob, t):
    """Dxx, Dxy, Dyy from a D table at the cell centres: bilinear in alpha0 and log E between its
    end points, the end nodes beyond them, then the conversion of units."""
    x, y = 0.5 * (prob.x_edges[:-1] + prob.x_edges[1:]), 0.5 * (prob.y_edges[:-1] + prob.y_edges[1:])

    def where(v, lo, hi, n):
        pos = np.clip((v - lo) / (hi - lo) * (n - 1), 0.0, n - 1)
        k = np.minimum(pos.astype(int), n - 2)
        return k, pos - k

    ia, u = where(x, np.radians(t.alpha0_deg[0]), np.radians(t.alpha0_deg[-1]), len(t.alpha0_deg))
    je, w = where(y, math.log(t.E[0]), math.log(t.E[-1]), len(t.E))
    u, w = u[:, None], w[None, :]

    def at(T):
        c = lambda a, b: T[np.ix_(ia + a, je + b)]
        return (1 - u) * (1 - w) * c(0, 0) + u * (1 - w) * c(1, 0) + u * w * c(1, 1) + (1 - u) * w * c(0, 1)

    e0 = 0.511875
    E = np.exp(y)
    p = np.sqrt(E * (E + 2 * e0))
    dl = p / (E * (E + e0))
    k = e0 * e0 * 86400.0
    return at(t.Daa) * k / (p * p), at(t.Dap) * k * dl / p, at(t.Dpp) * k * dl * dl


def exact(case, seed):
    form = case["form"]
    if form == "server":
        reqs = sorted(enumerate(_requests(case, seed)), key=lambda q: (-q[1][0].nx, q[0]))
        got = [None] * len(reqs)
        for at in range(0, len(reqs), 8):  # requests of similar grids together
            part = reqs[at:at + 8]
            left = dict(enumerate(part))
            ex = _Exact([p for _, (p, _) in part], [(p.Dxx, p.Dxy, p.Dyy) for _, (p, _) in part])
            for n in range(1, max(s for _, (_, s) in part) + 1):
                ex.step()
                for k, (r, (_, s)) in left.items():
                    if s == n:
                        got[r] = ex.get(k).ravel()
        return np.concatenate(got)
    if form == "host":
        probs, which = _batch_problems(case, seed)
        fields = [(p.Dxx, p.Dxy, p.Dyy) for p in probs]
    else:
        prob, table = _problem(case, seed)
        probs, which = [prob], [0]
        fields = [(prob.Dxx, prob.Dxy, prob.Dyy) if table is None else _table_fields(prob, table)]
    ex = _Exact(probs, fields)
    for _ in range(case["steps"]):
        ex.step()
    got = [ex.get(k) for k in range(len(probs))]
    if form == "host":
        return torch.from_numpy(np.concatenate([got[k].ravel() for k in which]))
    if form == "noalloc":
        return torch.tensor(got[0])
    return got[0]
