"""The work that users of the library have it do, as measurable cases.

A case is one pass through the public entry points (`Simp`, `Batch`, `Server`) on a seeded
synthetic basin.  What each kind of case stands for:

  run      a basin resident on the GPU advanced to its next output time: `steps` steps of the
           time loop, then the state read back (the drop-in time_integration of the Fortran host)
  rates    one right-hand side for a host that keeps its own integrator: the state handed over,
           the rates read back (the drop-in single_step)
  coupled  a host that owns the state and exchanges it every step: upload, one step enqueued,
           read back
  pairs    the neighbour search alone: the sorted pair lists with their distances
  batch    an ensemble of uneven basins advanced together, every member read back
  served   a stream of requests of uneven sizes and step counts through the serving loop

and each set of switches (`physics`):

  basin       cubic spline, hsml = 2.4 dx held, fixed dt, walls and uniform wind: the synthetic
              basins of this repository (FP64, or mixed precision)
  vortex      the same under a cyclonic vortex with walls all around
  reference   the values the reference ships: Wendland C6, hsml = 3 sqrt(m / rho) evolving, the
              viscous-plastic time step
  continuity  Gaussian kernel, continuity density, XSPH and Monaghan's artificial viscosity

Basins are in motion (a smooth velocity field) with thickness and concentration that vary over
the basin, on a jittered lattice whose last row may be ragged, and fixed time steps lie under the
viscous-plastic bound.
"""
import math

import numpy as np
import torch

from simp_b200 import basins, serve
from simp_b200.params import ART_VISC_MON, PREC_FP64, PREC_MIXED, SKF_GAUSSIAN, reference_default
from simp_b200.simp import Batch, Simp

KINDS = ("run", "rates", "coupled", "pairs", "batch", "served")
PHYSICS = ("basin", "vortex", "reference", "continuity")


def listed():
    return [
        # one step and its read-back on a coarse regional basin: launches and waits
        {"name": "step_1024", "kind": "run", "physics": "basin", "mixed": False, "n": 1024, "dx": 2000.0,
         "steps": 1},
        # the smallest of the repository's workloads, its time loop to an output
        {"name": "run_2500", "kind": "run", "physics": "basin", "mixed": False, "n": 2500, "dx": 2000.0,
         "steps": 200},
        # a medium basin of odd size in mixed precision
        {"name": "run_24649_mixed", "kind": "run", "physics": "basin", "mixed": True, "n": 24649, "dx": 1000.0,
         "steps": 100},
        # the headline basin: 512 x 512 at 500 m, FP64
        {"name": "run_262144", "kind": "run", "physics": "basin", "mixed": False, "n": 262144, "dx": 500.0,
         "steps": 100},
        # the largest single basin: 1024 x 1024 at 250 m under a vortex, mixed precision
        {"name": "run_1048576_mixed", "kind": "run", "physics": "vortex", "mixed": True, "n": 1048576, "dx": 250.0,
         "steps": 60},
        # a large ragged basin in plain FP64
        {"name": "run_600011", "kind": "run", "physics": "vortex", "mixed": False, "n": 600011, "dx": 500.0,
         "steps": 40},
        # the switches the reference ships, on a basin of its own resolution
        {"name": "run_reference_90007", "kind": "run", "physics": "reference", "mixed": False, "n": 90007,
         "dx": 2000.0, "steps": 60},
        # the regularised form with continuity density
        {"name": "run_continuity_40401", "kind": "run", "physics": "continuity", "mixed": False, "n": 40401,
         "dx": 2000.0, "steps": 60},
        # a host integrator asking for one right-hand side of its state
        {"name": "rates_65025", "kind": "rates", "physics": "basin", "mixed": False, "n": 65025, "dx": 1000.0,
         "steps": 1},
        # the neighbour search on its own
        {"name": "pairs_50003", "kind": "pairs", "physics": "basin", "mixed": False, "n": 50003, "dx": 1000.0,
         "steps": 1},
        # eight uneven basins, log-uniform in size as the ensemble's, in mixed precision
        {"name": "batch_8_mixed", "kind": "batch", "physics": "basin", "mixed": True, "n": 262144, "count": 8,
         "dx": 1000.0, "steps": 60},
        # twelve requests of uneven size and length through the server, in mixed precision
        {"name": "served_12_mixed", "kind": "served", "physics": "basin", "mixed": True, "n": 131072, "count": 12,
         "dx": 1000.0, "steps": 200},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("run", "run", "run", "run", "rates", "coupled", "pairs", "batch", "served"))
    physics = rng.choice(PHYSICS) if kind == "run" else "basin"
    mixed = physics in ("basin", "vortex") and kind in ("run", "batch", "served") and rng.random() < 0.5
    c = {"kind": kind, "physics": physics, "mixed": mixed, "dx": rng.choice((250.0, 500.0, 1000.0, 2000.0)),
         "steps": 1}
    if kind == "run":
        c["n"] = _log_uniform(rng, 1024, 1048576 if physics in ("basin", "vortex") else 131072)
        c["steps"] = _log_uniform(rng, 1, max(2, min(200, 60 * 1048576 // (3 * c["n"]))))
    elif kind in ("batch", "served"):
        c["mixed"] = c["mixed"] or kind == "served"
        c["n"] = _log_uniform(rng, 16384, 262144 if kind == "batch" else 131072)
        c["count"] = rng.randint(3, 8 if kind == "batch" else 12)
        c["steps"] = _log_uniform(rng, 4, 60 if kind == "batch" else 200)
    else:
        c["n"] = _log_uniform(rng, 1024, 131072)
    return c


# --- inputs ------------------------------------------------------------------

def _smooth(x, L, rng, lo, hi):
    """A smooth field over the basin with values in (lo, hi)."""
    k = 2.0 * np.pi / L
    p = rng.uniform(0.0, 2.0 * np.pi, size=4)
    f = 0.25 * (np.sin(2 * k * x[:, 0] + p[0]) + np.cos(3 * k * x[:, 1] + p[1])
                + np.sin(k * (x[:, 0] + x[:, 1]) + p[2]) + np.cos(k * (x[:, 0] - 2 * x[:, 1]) + p[3]))
    return 0.5 * (lo + hi) + 0.5 * (hi - lo) * f


def _basin(case, n, seed, walls="+x-x+y-y"):
    """A basin of exactly n particles: the first n of the smallest square lattice that holds them."""
    rng = np.random.default_rng(seed)
    dx = case["dx"]
    nside = max(2, math.isqrt(n - 1) + 1)
    L = nside * dx
    ang, speed = rng.uniform(0.0, 2.0 * np.pi), rng.uniform(5.0, 15.0)
    vortex = None
    if case["physics"] == "vortex":
        vortex = (rng.uniform(0.25, 0.75) * L, rng.uniform(0.25, 0.75) * L, 15.0, 0.1 * L)
    b = basins.make_basin(nside, dx, int(rng.integers(1 << 31)), walls=walls,
                          wind=(speed * math.cos(ang), speed * math.sin(ang)), vortex=vortex,
                          precision=PREC_MIXED if case["mixed"] else PREC_FP64)
    b.x = np.ascontiguousarray(b.x[:n])
    b.vx = basins.smooth_velocity(b.x, L, amp=0.3, seed=int(rng.integers(1 << 31)))
    b.h = _smooth(b.x, L, rng, 0.5, 2.0)
    b.A = _smooth(b.x, L, rng, 0.8, 1.0)
    b.rho = 900.0 * b.h
    b.mass = b.rho * dx * dx
    b.hsml = np.ascontiguousarray(b.hsml[:n])
    b.massb = np.full(b.nb, b.mass.mean())
    p = b.params
    # a third of the viscous-plastic bound rho_ice hsml^2 delta_min / P_star at h = 1
    p.dt = basins.vp_dt_bound(dx) / 6.0
    if case["physics"] == "reference":
        q = reference_default()
        q.wind_u, q.wind_v, q.b_length = p.wind_u, p.wind_v, p.b_length
        b.hsml = np.full(n, 3.0 * dx)
        q.dt = q.rho_ice * (3.0 * dx) ** 2 * q.delta_min / (q.P_star * (1.0 + q.k_t))
        b.params = q
    elif case["physics"] == "continuity":
        p.skf, p.den_alg = SKF_GAUSSIAN, 2
        p.xsph_regularization, p.artificial_visc, p.art_visc_alg = 1, 1, ART_VISC_MON
    return b


def _walls(case):
    """Sides with walls: none for the search alone (open water), one or four for a basin."""
    if case["kind"] == "pairs":
        return ""
    return "+x" if case["physics"] in ("basin", "continuity") else "+x-x+y-y"


def _sizes(case):
    """Sizes (log-uniform up to n) and, for a stream, step counts of several basins."""
    rng = np.random.default_rng(case["n"] + 100 * case["steps"])
    lo = 4096 if case["kind"] == "batch" else 1024
    n = np.exp(rng.uniform(math.log(lo), math.log(case["n"]), size=case["count"] - 1))
    steps = rng.integers(max(1, case["steps"] // 20), case["steps"] + 1, size=case["count"])
    return [case["n"]] + [int(v) for v in n], [int(v) for v in steps]


def _many(case, seed):
    sizes, steps = _sizes(case)
    return [_basin(case, n, 1000 * seed + k) for k, n in enumerate(sizes)], steps


def prepare(case, seed):
    if case["kind"] in ("batch", "served"):
        bs, steps = _many(case, seed)
        nb = sum(b.nb for b in bs)
        if case["kind"] == "batch":
            batch = Batch(bs[0].params, sum(b.n for b in bs), nb, len(bs))
            return {"case": case, "batch": batch, "slots": [batch.add(b) for b in bs]}
        requests = [serve.Request(b, k, 0.0) for b, k in zip(bs, steps)]
        server = serve.Server(bs[0].params, 4.0e9, max_instances=32, max_request_particles=case["n"])
        return {"case": case, "server": server, "requests": requests}
    b = _basin(case, case["n"], seed, _walls(case))
    return {"case": case, "basin": b, "sim": Simp.from_basin(b)}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        state["batch"].step(case["steps"])
        return [state["batch"].get_state(s) for s in state["slots"]]
    if kind == "served":
        server = state["server"]
        ids = [server.submit(r) for r in state["requests"]]
        server.run()
        return [server.outputs.pop(i) for i in ids]
    sim, b = state["sim"], state["basin"]
    if kind == "run":
        sim.time_integration(case["steps"])
        return sim.get_state()
    if kind == "pairs":
        return sim.nnps()
    sim.set_state(b.x, b.vx, b.mass, b.rho, b.hsml, b.A, b.h, b.xb, b.massb, b.params.dt, 60.0)
    if kind == "rates":
        return sim.single_step(60.0)
    sim.step_enqueue(1)
    return sim.get_state()


def work(case):
    """Bytes and FP64 operations a pass cannot do without.

    Per particle and step 704 B (two right-hand sides: search 24 B, kinematic 88 B, stress 136 B,
    update 104 B) and, per pair seen from one side, about 60 operations in the kinematic and 45 in
    the stress sums; each read-back or upload moves the particle's 9 doubles once more.
    """
    pairs = 28 if case["physics"] == "reference" else 20
    rhs = 2.0 * pairs * 105 + 200.0
    if case["kind"] in ("batch", "served"):
        # (sizes log-uniform between lo and n: their mean)
        lo = 4096.0 if case["kind"] == "batch" else 1024.0
        mean = (case["n"] - lo) / math.log(case["n"] / lo)
        n = case["n"] + (case["count"] - 1) * mean
        steps = case["steps"] * (1.0 if case["kind"] == "batch" else 0.525)
    else:
        n, steps = float(case["n"]), float(case["steps"])
    if case["kind"] == "pairs":
        return {"bytes": n * (24.0 + 12.0 * 0.5 * pairs * 2), "flops": n * pairs * 8.0}
    if case["kind"] == "rates":
        return {"bytes": n * (248.0 + 72.0 + 48.0), "flops": n * rhs / 2}
    return {"bytes": n * (704.0 * steps + 72.0 * (2 if case["kind"] == "coupled" else 1)), "flops": n * rhs * steps}


# --- the same in plain 64-bit torch --------------------------------------------

_DEV = "cuda" if torch.cuda.is_available() else "cpu"
_WALL_DEN = {"cubic": 2.0, "wendland_c6": 1.0, "gaussian": 3.0}   # scale_h of each kernel


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=_DEV)


def _candidates(px, py, qx, qy, reach, drop_self):
    """Index pairs (i, j) with |p_i - q_j| <= reach, by cells of side reach, sorted by (i, j)."""
    x0, y0 = torch.minimum(px.min(), qx.min()) - 2 * reach, torch.minimum(py.min(), qy.min()) - 2 * reach
    ncx = int((torch.maximum(px.max(), qx.max()) - x0) / reach) + 3
    cq = ((qy - y0) / reach).long() * ncx + ((qx - x0) / reach).long()
    order = torch.argsort(cq, stable=True)
    ncells = (int((torch.maximum(py.max(), qy.max()) - y0) / reach) + 3) * ncx
    count = torch.bincount(cq, minlength=ncells)
    start = torch.cumsum(count, 0) - count
    cp = ((py - y0) / reach).long() * ncx + ((px - x0) / reach).long()
    rows = torch.arange(px.numel(), device=px.device)
    out_i, out_j = [], []
    for dy in (-1, 0, 1):
        for dxc in (-1, 0, 1):
            c = cp + dy * ncx + dxc
            a, m = start[c], count[c]
            for k in range(int(m.max())):
                has = m > k
                i, j = rows[has], order[(a + k)[has]]
                near = (px[i] - qx[j]) ** 2 + (py[i] - qy[j]) ** 2 <= reach * reach
                if drop_self:
                    near &= i != j
                out_i.append(i[near])
                out_j.append(j[near])
    i, j = torch.cat(out_i), torch.cat(out_j)
    o = torch.argsort(i * max(1, qx.numel()) + j)
    return i[o], j[o]


class _Exact:
    """One basin of the reference's scheme in plain 64-bit torch."""

    def __init__(self, b):
        self.p = b.params
        self.kernel = {9: "cubic", 6: "wendland_c6", 2: "gaussian"}[self.p.skf]
        self.x, self.y = _t(b.x[:, 0]), _t(b.x[:, 1])
        self.u, self.v = _t(b.vx[:, 0]), _t(b.vx[:, 1])
        self.m, self.rho, self.hs, self.A, self.h = (_t(a) for a in (b.mass, b.rho, b.hsml, b.A, b.h))
        self.xb, self.yb, self.mb = _t(b.xb[:, 0]), _t(b.xb[:, 1]), _t(b.massb)
        self.max_hs = self.p.max_hsml if self.p.max_hsml > 0 else 10.0 * float(self.hs.max())
        self.dt, self.t = float(self.p.dt), 0.0
        self.lists_at = None

    # W and f with grad W = f (x_i - x_j); sh r / h = q
    def _w(self, r, h):
        if self.kernel == "cubic":
            s, q = 2.0 / h, 2.0 * r / h
            f = 15.0 / (7.0 * math.pi) * s * s
            two_thirds, sixth = float(np.float32(2.0 / 3.0)), float(np.float32(1.0 / 6.0))
            near = q <= 1.0
            w = torch.where(near, two_thirds - q * q + 0.5 * q ** 3, sixth * (2.0 - q) ** 3)
            g = torch.where(near, 1.5 * q * q - 2.0 * q, -0.5 * (2.0 - q) ** 2)
        elif self.kernel == "wendland_c6":
            s, q = 1.0 / h, r / h
            f = 78.0 / (7.0 * math.pi) * s * s
            w = (1.0 - q) ** 8 * (32.0 * q ** 3 + 25.0 * q * q + 8.0 * q + 1.0)
            g = -22.0 * q * (1.0 - q) ** 7 * (16.0 * q * q + 7.0 * q + 1.0)
        else:
            s, q = 3.0 / h, 3.0 * r / h
            f = 1.0 / math.pi * s * s
            w = torch.exp(-q * q)
            g = -2.0 * q * w
        return f * w, f * g * s / r

    def _wall_w(self, d, hs):
        bl = self.p.b_length
        if self.kernel == "wendland_c6":
            q = d / bl
            return 78.0 / (7.0 * math.pi) / (hs * hs) * (1.0 - q) ** 8 * (32.0 * q ** 3 + 25.0 * q * q + 8.0 * q + 1.0)
        sh = _WALL_DEN[self.kernel]
        q, f = d / bl * sh, (sh / bl) ** 2
        if self.kernel == "gaussian":
            return f / math.pi * torch.exp(-q * q)
        two_thirds, sixth = float(np.float32(2.0 / 3.0)), float(np.float32(1.0 / 6.0))
        return 15.0 / (7.0 * math.pi) * f * torch.where(
            q <= 1.0, two_thirds - q * q + 0.5 * q ** 3, torch.where(q <= 2.0, sixth * (2.0 - q) ** 3, torch.zeros_like(q)))

    def _lists(self, x, y, hs):
        reach = 1.1 * float(hs.max())
        if self.lists_at is not None:
            x0, y0, had = self.lists_at
            moved = float(torch.sqrt(((x - x0) ** 2 + (y - y0) ** 2).max()))
            if float(hs.max()) + 2.0 * moved <= had:
                return
        self.lists_at = (x.clone(), y.clone(), reach)
        self.ci, self.cj = _candidates(x, y, x, y, reach, True)
        self.wi = self.wj = None
        if self.xb.numel():
            self.wi, self.wj = _candidates(x, y, self.xb, self.yb, self.p.b_length + 0.1 * reach, False)

    def pairs(self, x, y, hs):
        self._lists(x, y, hs)
        i, j = self.ci, self.cj
        r = torch.sqrt((x[i] - x[j]) ** 2 + (y[i] - y[j]) ** 2)
        hij = (hs[i] + hs[j]) / 2.0
        k = r <= hij
        return i[k], j[k], r[k], hij[k]

    def _sum(self, i, v, n):
        return torch.zeros(n, dtype=torch.float64, device=_DEV).index_add_(0, i, v)

    def _sound(self, rho):
        return torch.sqrt(self.p.Y * (1.0 - self.p.nu) / (rho * (1.0 + self.p.nu) * (1.0 - 2.0 * self.p.nu)))

    def rhs(self, x, y, u, v, m, rho, hs, A, h, t):
        """dx/dt, dv/dt, dh/dt, dA/dt, the divergence sum, and the pairs with their gradients."""
        p, n = self.p, x.numel()
        i, j, r, hij = self.pairs(x, y, hs)
        dx, dy, du, dv = x[i] - x[j], y[i] - y[j], u[i] - u[j], v[i] - v[j]
        w, f = self._w(r, hij)
        gx, gy = f * dx, f * dy
        mj, mr = m[j], m[j] / rho[j]
        div = -self._sum(i, mj * (du * gx + dv * gy), n)
        e11, e22 = -self._sum(i, mr * du * gx, n), -self._sum(i, mr * dv * gy, n)
        e12 = -0.5 * self._sum(i, mr * (dv * gx + du * gy), n)
        em2 = 1.0 / (p.e * p.e)
        strength = p.P_star * h * torch.exp(-p.c_eos * (1.0 - A))
        delta = torch.sqrt((e11 ** 2 + e22 ** 2) * (1.0 + em2) + 4.0 * em2 * e12 ** 2 + 2.0 * e11 * e22 * (1.0 - em2))
        zeta = 0.5 * strength * (1.0 + p.k_t) / torch.clamp(delta, min=p.delta_min)
        eta = zeta / (p.e * p.e)
        pr = 2.0 * zeta * delta / (1.0 + p.k_t) * (1.0 - p.k_t) / 2.0
        r2 = rho * rho
        t11 = ((zeta + eta) * e11 + (zeta - eta) * e22 - pr) / r2
        t22 = ((zeta + eta) * e22 + (zeta - eta) * e11 - pr) / r2
        t12 = 2.0 * eta * e12 / r2
        fi = rho / p.rho_ice / h
        ax = fi * self._sum(i, mj * ((t11[i] + t11[j]) * gx + (t12[i] + t12[j]) * gy), n)
        ay = fi * self._sum(i, mj * ((t12[i] + t12[j]) * gx + (t22[i] + t22[j]) * gy), n)
        if self.wi is not None:
            bdx, bdy = self.xb[self.wj] - x[self.wi], self.yb[self.wj] - y[self.wi]
            d = torch.sqrt(bdx * bdx + bdy * bdy)
            k = d <= p.b_length
            wi, wj, d, bdx, bdy = self.wi[k], self.wj[k], d[k], bdx[k], bdy[k]
            c = p.kappa_n * self._wall_w(d, hs[wi]) * 2.0 * self.mb[wj] / ((m[wi] + self.mb[wj]) * d * d)
            ax = ax - self._sum(wi, c * bdx, n) / rho
            ay = ay - self._sum(wi, c * bdy, n) / rho
        if t > 0.0:
            if p.wind_kind == 1:
                rx, ry = x - p.vortex_x, y - p.vortex_y
                rr = torch.sqrt(rx * rx + ry * ry)
                s = rr / p.vortex_radius
                U = p.vortex_umax * s * torch.exp(0.5 * (1.0 - s * s))
                wu, wv = -U * ry / rr, U * rx / rr
            else:
                wu, wv = p.wind_u, p.wind_v
            ka, kw = p.c_wind * p.rho_air / (h * p.rho_ice), p.c_water * p.rho_water / (h * p.rho_ice)
            ax = ax + ka * (wu - u) * torch.abs(wu - u) + kw * (p.current_u - u) * torch.abs(p.current_u - u)
            ay = ay + ka * (wv - v) * torch.abs(wv - v) + kw * (p.current_v - v) * torch.abs(p.current_v - v)
        xt, yt = u, v
        if p.xsph_regularization:
            rbar = 0.5 * (rho[i] + rho[j])
            xt = u - p.chi * self._sum(i, mj * du * w / rbar, n)
            yt = v - p.chi * self._sum(i, mj * dv * w / rbar, n)
        if p.artificial_visc:
            vr = du * dx + dv * dy
            cor = float(np.float32(0.01)) * hij
            iota = hij * vr / (r * r + cor * cor)
            c = self._sound(rho)
            pi = (p.beta_pi * iota * iota - p.alpha_pi * iota * (c[i] + c[j]) / 2.0) / ((rho[i] + rho[j]) / 2.0)
            pi = torch.where(vr <= 0.0, pi, torch.zeros_like(pi))
            ax = ax - self._sum(i, mj * pi * gx, n)
            ay = ay - self._sum(i, mj * pi * gy, n)
        return xt, yt, ax, ay, -h * div / rho, -A * div / rho, div, (i, j, gx, gy)

    def step(self):
        p, dt, n = self.p, self.dt, self.x.numel()
        s = (self.x, self.y, self.u, self.v)
        xt, yt, ax, ay, ht, At, div, (i, j, gx, gy) = self.rhs(*s, self.m, self.rho, self.hs, self.A, self.h, self.t)
        x, y = self.x + xt * dt / 2.0, self.y + yt * dt / 2.0
        u, v = self.u + ax * dt / 2.0, self.v + ay * dt / 2.0
        h, A = self.h + ht * dt / 2.0, torch.clamp(self.A + At * dt / 2.0, max=1.0)
        if p.den_alg == 2:
            drho = self._sum(i, self.m[j] * ((u[i] - u[j]) * gx + (v[i] - v[j]) * gy), n)
            rho = self.rho + drho * dt / 2.0
        else:
            rho = h * p.rho_ice
        xt, yt, ax, ay, ht, At, div, _ = self.rhs(x, y, u, v, self.m, rho, self.hs, A, h, self.t)
        self.x, self.y = self.x + xt * dt, self.y + yt * dt
        self.u, self.v = self.u + ax * dt, self.v + ay * dt
        self.h, self.A = self.h + ht * dt, torch.clamp(self.A + At * dt, max=1.0)
        self.rho = self.rho - div * dt if p.den_alg == 2 else self.h * p.rho_ice
        if p.sle == 2:
            self.hs = torch.clamp(torch.sqrt(self.m / self.rho) * p.hsml_multiplicity, max=self.max_hs)
        if p.tse == 2:
            self.dt = float((p.rho_ice * self.hs * self.hs * p.delta_min / (p.P_star * (1.0 + p.k_t))).min())
        self.t += self.dt

    def state(self, keys=("x", "vx", "mass", "rho", "hsml", "A", "h", "dt", "current_time")):
        out = {"x": torch.stack((self.x, self.y), 1), "vx": torch.stack((self.u, self.v), 1), "mass": self.m,
               "rho": self.rho, "hsml": self.hs, "A": self.A, "h": self.h, "dt": self.dt, "current_time": self.t}
        return {k: out[k].cpu().numpy() if isinstance(out[k], torch.Tensor) else out[k] for k in keys}


def _advance(b, steps):
    e = _Exact(b)
    for _ in range(steps):
        e.step()
    return e


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        bs, _ = _many(case, seed)
        keys = ("x", "vx", "mass", "rho", "hsml", "A", "h", "current_time")
        return [_advance(b, case["steps"]).state(keys) for b in bs]
    if kind == "served":
        bs, steps = _many(case, seed)
        return [_advance(b, k).state(("x", "vx", "h", "A")) for b, k in zip(bs, steps)]
    b = _basin(case, case["n"], seed, _walls(case))
    if kind == "run":
        return _advance(b, case["steps"]).state()
    e = _Exact(b)
    if kind == "pairs":
        i, j, r, hij = e.pairs(e.x, e.y, e.hs)
        k = i < j
        return {"nip": None, "p_i": None, "p_j": None, "r_ij": r[k].cpu().numpy(), "hsml_ij": hij[k].cpu().numpy(),
                "bnip": None, "bp_i": None, "bp_j": None, "br_ij": None}
    e.t = 60.0
    if kind == "coupled":
        e.step()
        return e.state()
    xt, yt, ax, ay, ht, At, _, _ = e.rhs(e.x, e.y, e.u, e.v, e.m, e.rho, e.hs, e.A, e.h, 60.0)
    out = {"dxdt": torch.stack((xt, yt), 1), "dvxdt": torch.stack((ax, ay), 1), "dhdt": ht, "dAdt": At}
    return {k: v.cpu().numpy() for k, v in out.items()}
