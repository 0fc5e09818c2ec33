"""Performance cases: the SPH workloads that programs run through the C ABI.

A pass is what a caller that owns the particle state does between two of its
own frames (the Go shim's Sync, the end-to-end leg of bench.py): hand the
state over (sph_set_state), advance it some steps (sph_step), read the state
and the derived fields back (sph_get_state, sph_get_derived), and for an
animation draw the frame (sph_render). Every pass starts from the same state,
two steps into the run. One case calls the allocation-free density instead.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

STATE = ("x", "y", "vx", "vy", "u", "ax", "ay", "udot")
DERIVED = ("rho", "c", "h")
PREP_STEPS = 2           # steps between the initial condition and a pass's state
DBL_MAX = np.finfo(np.float64).max
OPEN = (-DBL_MAX, DBL_MAX)
GRAVITY = (0.0, 0.5)
TANK = (0.1, 0.9, 0.1, 0.9)
FRAME = (1280, 720)      # the animator's canvas
EXACT_MAX_N = 140_000    # larger runs take the plain restatement too long


def case(name, kind, n, k, form, steps, kernel="Monahan", level=0, sims=1, frame=False):
    return {"name": name, "kind": kind, "n": n, "k": k, "form": form, "steps": steps, "kernel": kernel,
            "level": level, "sims": sims, "frame": frame}


def listed():
    return [
        # the reference's default simulation: one rectangle of 1000 particles, open bounds
        case("rect 1000 open exact", "rect", 1000, 32, "Exact", 10),
        # the smallest benchmark workload, as a drop-in and in the mixed form
        case("blast 10k exact", "blast", 10_000, 32, "Exact", 10),
        case("blast 10k mixed", "blast", 10_000, 32, "Mixed", 10),
        # the speed test's particle count, with the frame its animator draws
        case("speed test 100k frame", "blast", 100_000, 32, "Exact", 4, frame=True),
        # a walled tank under gravity: open axes, reflections, Wendland kernel, ragged n and k
        case("tank 65537 k21 wendland", "tank", 65_537, 21, "Exact", 4, kernel="Wendland"),
        # the blast wave at scale
        case("blast 1M exact", "blast", 1_048_576, 32, "Exact", 2),
        case("blast 1M mixed", "blast", 1_048_576, 32, "Mixed", 6),
        # the headline workload: 64 blobs over a background, radii varying about tenfold
        case("clustered 4M exact", "clustered", 4_194_304, 32, "Exact", 2),
        case("clustered 4M mixed", "clustered", 4_194_304, 32, "Mixed", 6),
        # nearly everything in a hundredth of the box, long lists, an explicit grid level
        case("stress 2M k64 exact", "stress", 2_000_003, 64, "Exact", 2, level=13),
        # many small simulations advanced together
        case("ensemble 48 exact", "ensemble", 5, 32, "Exact", 4, sims=48),
        # one density query of a latency-bound caller that may not allocate
        case("noalloc 4096", "noalloc", 4096, 32, "Exact", 1),
    ]


def log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def auto_level(n):
    return int(min(max(math.floor(0.5 * math.log2(max(n, 2) / 2.0) + 0.5), 1), 14))


def draw(rng):
    kind = rng.choice(["blast", "blast", "clustered", "clustered", "rect", "tank", "stress", "ensemble", "noalloc"])
    form = rng.choice(["Exact", "Exact", "Mixed", "Mixed", "Fast"])
    k = rng.choice([32, 32, 32, 16, 21, 24, 48, 64])
    kernel = rng.choice(["Monahan", "Monahan", "Wendland"])
    level, sims, frame, steps = 0, 1, False, rng.randint(2, 6)
    if kind == "noalloc":
        n, form, k, steps = log_int(rng, 700, 8192), "Exact", rng.choice([32, 16, 21, 24]), 1
    elif kind == "ensemble":
        n, sims = rng.randint(1, 1 << 20), rng.randint(8, 64)  # n seeds the member sizes
    elif kind in ("rect", "tank"):
        n, frame = log_int(rng, 1000, 300_000), rng.random() < 0.3
    elif kind == "stress":
        n = log_int(rng, 60_000, 1_500_000)
        level = min(auto_level(n) + 3, 14)
    else:
        n = log_int(rng, 1000, 2_500_000)
    if kind not in ("noalloc", "ensemble") and rng.random() < 0.7:
        n |= 1
    c = case("", kind, n, k, form, steps, kernel, level, sims, frame)
    del c["name"]
    return c


# ------------------------------------------------------------------- inputs
def sizes(case):
    """Particle counts of the simulations of a case (an ensemble's are log-uniform in [1000, 65536])."""
    if case["kind"] != "ensemble":
        return [case["n"]]
    r = np.random.default_rng(case["n"])
    return [int(v) for v in np.exp(r.uniform(math.log(1000.0), math.log(65536.0), case["sims"]))]


def flow(x, y, rng, amp):
    """A smooth periodic velocity field (a few Fourier modes)."""
    p = rng.uniform(0.0, 2 * np.pi, 4)
    t = 2 * np.pi
    return (amp * (np.sin(t * y + p[0]) + 0.5 * np.sin(t * (2 * x - y) + p[1])),
            amp * (np.sin(t * x + p[2]) + 0.5 * np.sin(t * (x + 2 * y) + p[3])))


def initial(case, n, rng):
    """(x, y, vx, vy, u) of one simulation."""
    kind = case["kind"]
    if kind in ("clustered",):
        nb = 64
        cx, cy = rng.random(nb), rng.random(nb)
        sig = np.exp(rng.uniform(math.log(0.005), math.log(0.05), nb))
        nbg = n // 5
        b = rng.integers(0, nb, n)
        gx, gy = rng.standard_normal(n), rng.standard_normal(n)
        x, y = cx[b] + sig[b] * gx, cy[b] + sig[b] * gy
        x, y = x - np.floor(x), y - np.floor(y)
        core = gx * gx + gy * gy < 1.0
        x[:nbg], y[:nbg], core[:nbg] = rng.random(nbg), rng.random(nbg), False
        x[x >= 1.0], y[y >= 1.0] = 0.0, 0.0
        u = np.where(core, 10.0, 1.0)
    elif kind == "stress":
        ox, oy = rng.uniform(0.0, 0.9, 2)
        x, y = rng.random(n), rng.random(n)
        m = n - n // 100
        x[:m], y[:m] = ox + 0.1 * x[:m], oy + 0.1 * y[:m]
        u = np.where((x - ox - 0.05) ** 2 + (y - oy - 0.05) ** 2 < 1e-4, 100.0, 1.0)
    elif kind == "rect":
        x, y = rng.random(n), rng.random(n)
        return x, y, np.zeros(n), np.zeros(n), np.full(n, 0.01)
    elif kind == "tank":
        x = TANK[0] + (TANK[1] - TANK[0]) * rng.random(n)
        y = TANK[2] + (TANK[3] - TANK[2]) * rng.random(n)
        u = np.where((x - 0.5) ** 2 + (y - 0.5) ** 2 < 0.01, 3.0, 1.0)
    else:
        x, y = rng.random(n), rng.random(n)
        hot = rng.uniform(5.0, 50.0) if kind == "ensemble" else 10.0
        u = np.where((x - 0.5) ** 2 + (y - 0.5) ** 2 < 0.01, hot, 1.0)
    vx, vy = flow(x, y, rng, 0.3)
    return x, y, vx, vy, u


def time_step(case, n):
    s = {"clustered": 5e-3, "stress": 1e-3, "rect": 6e-2, "tank": 1e-2, "blast": 1e-2, "ensemble": 5e-3,
         "noalloc": 1e-2}[case["kind"]]
    return s / math.sqrt(n)


def settings(case, n):
    """Physics of one simulation, as plain values."""
    p = {"k": case["k"], "kernel": case["kernel"], "gamma": 5.0 / 3.0, "mass": 1.0 / n, "dth": time_step(case, n) / 2,
         "accel": (0.0, 0.0), "hor": (0.0, 1.0), "vert": (0.0, 1.0), "refl": OPEN + OPEN,
         "alpha": 1.0, "beta": 2.0, "etasq": 0.01}
    if case["kind"] == "rect":    # the reference's constants and defaults
        p |= {"gamma": 1.66666, "mass": 1.0, "hor": OPEN, "vert": OPEN, "alpha": 0.75, "beta": 1.5}
    elif case["kind"] == "tank":
        p |= {"accel": GRAVITY, "hor": OPEN, "vert": OPEN, "refl": TANK}
    return p


def inputs(case, seed):
    """[(settings, (x, y, vx, vy, u))] of the case's simulations."""
    rng = np.random.default_rng(seed)
    return [(settings(case, n), initial(case, n, rng)) for n in sizes(case)]


# -------------------------------------------------------------------- runs
def sph_params(case, p):
    from sphugo_gb300 import _lib as L

    q = L.load().sph_default_params()
    q.k, q.grid_level = p["k"], case["level"]
    q.kernel = L.KERNEL_WENDLAND if p["kernel"] == "Wendland" else L.KERNEL_MONAHAN
    q.precision = {"Exact": L.PREC_FP64, "Mixed": L.PREC_MIXED, "Fast": L.PREC_FP64_FAST}[case["form"]]
    q.gamma, q.mass, q.dth = p["gamma"], p["mass"], p["dth"]
    q.accel[:], q.hor[:], q.vert[:], q.refl[:] = p["accel"], p["hor"], p["vert"], p["refl"]
    q.alpha, q.beta, q.etasq = p["alpha"], p["beta"], p["etasq"]
    return q


def dptr(t):
    return C.cast(t.data_ptr(), C.POINTER(C.c_double))


class Stepper:
    """A simulation (or ensemble) handle with the caller's pinned host buffers."""

    def __init__(self, case, seed):
        from sphugo_gb300 import _lib as L

        self.L, self.lib, self.case = L, L.load(), case
        self.handle = C.c_void_p()
        sims = inputs(case, seed)
        counts = np.array([len(a[0]) for _, a in sims], np.int64)
        n = int(counts.sum())
        if len(sims) == 1:
            p = sph_params(case, sims[0][0])
            L.check(self.lib.sph_create(C.byref(p), n, C.byref(self.handle)))
        else:
            ps = (L.SphParams * len(sims))(*[sph_params(case, p) for p, _ in sims])
            L.check(self.lib.sph_ens_create(ps, L.i64ptr(counts), len(sims), C.byref(self.handle)))
        cat = [np.ascontiguousarray(np.concatenate([a[i] for _, a in sims])) for i in range(5)]
        L.check(self.lib.sph_upload(self.handle, *[L.dptr(a) for a in cat]))
        L.check(self.lib.sph_step(self.handle, PREP_STEPS))
        buf = [torch.empty(n, dtype=torch.float64, pin_memory=True) for _ in range(19)]
        self.begin, self.end, self.derived = buf[:8], buf[8:16], buf[16:]
        L.check(self.lib.sph_get_state(self.handle, *[dptr(t) for t in self.begin]))
        self.out = dict(zip(STATE + DERIVED, self.end + self.derived))
        if case["frame"]:
            self.out["rgba"] = torch.empty((FRAME[1], FRAME[0], 4), dtype=torch.uint8, pin_memory=True)

    def run(self):
        L, lib, h = self.L, self.lib, self.handle
        L.check(lib.sph_set_state(h, *[dptr(t) for t in self.begin]))
        L.check(lib.sph_step(h, self.case["steps"]))
        L.check(lib.sph_get_state(h, *[dptr(t) for t in self.end]))
        L.check(lib.sph_get_derived(h, *[dptr(t) for t in self.derived]))
        if self.case["frame"]:
            L.check(lib.sph_render(h, *FRAME, C.cast(self.out["rgba"].data_ptr(), C.POINTER(C.c_uint8))))
        return self.out

    def __del__(self):
        if getattr(self, "handle", None):
            self.lib.sph_destroy(self.handle)


class NoAlloc:
    """A caller of the allocation-free density: device inputs and outputs."""

    def __init__(self, case, seed):
        from sphugo_gb300 import _lib as L

        self.L, self.lib = L, L.load()
        (p, arrays), = inputs(case, seed)
        self.n, k = case["n"], case["k"]
        self.p = sph_params(case, p)
        self.x, self.y = (torch.from_numpy(a).cuda() for a in arrays[:2])
        f = lambda m: torch.empty(m, dtype=torch.float64, device="cuda")  # noqa: E731
        self.out = {"ids": torch.empty(self.n * k, dtype=torch.int64, device="cuda"), "dist": f(self.n * k),
                    "rho": f(self.n), "h": f(self.n)}
        self.run()

    def run(self):
        o = self.out
        self.L.check(self.lib.sph_density_noalloc(
            C.byref(self.p), self.x.data_ptr(), self.y.data_ptr(), self.n, o["ids"].data_ptr(), o["dist"].data_ptr(),
            o["rho"].data_ptr(), o["h"].data_ptr(), torch.cuda.current_stream().cuda_stream or None))
        return o


def prepare(case, seed):
    return (NoAlloc if case["kind"] == "noalloc" else Stepper)(case, seed)


def run(state):
    return state.run()


def work(case):
    """Bytes: the caller's arrays in and out once. Flops: per neighbour and
    evaluation the density's 19 and the force's 24 (with 17 more for the half
    of the pairs that approach), an integration's 24 per particle."""
    n, k = sum(sizes(case)), case["k"]
    if case["kind"] == "noalloc":
        return {"bytes": n * (16 + 16 * k + 16), "flops": n * k * 13}
    frame = 4 * FRAME[0] * FRAME[1] if case["frame"] else 0
    return {"bytes": n * (64 + 88) + frame, "flops": case["steps"] * n * (k * (19 + 24 + 8.5) + 24)}


# ------------------------------------------- the same in plain 64-bit torch
def nearest(x, y, k, hor, vert):
    """(indices, dx, dy, d2), nearest first: image-shifted neighbour minus particle."""
    n = x.numel()
    periodic = hor != OPEN

    def offsets(i, j):
        dx, dy = x[j] - x[i], y[j] - y[i]
        return (dx - torch.round(dx), dy - torch.round(dy)) if periodic else (dx, dy)

    def pick(i, j, live):
        dx, dy = offsets(i, j)
        d2 = torch.where(live & (i != j), dx * dx + dy * dy, math.inf)
        v, o = torch.topk(d2, k, dim=1, largest=False)
        return torch.gather(j.expand_as(d2), 1, o), torch.gather(dx, 1, o), torch.gather(dy, 1, o), v

    every = torch.arange(n, device=x.device)

    def brute(q):
        chunk = max(1, (1 << 27) // n)
        got = [pick(c[:, None], every[None, :], torch.ones((), dtype=torch.bool, device=x.device))
               for c in torch.split(q, chunk)]
        return [torch.cat(t) for t in zip(*got)]

    if n <= 12_000:
        return brute(every)
    lo = torch.stack([x.min(), y.min()]) if not periodic else torch.zeros(2, dtype=x.dtype, device=x.device)
    size = float(torch.stack([x.max(), y.max()]).sub(lo).max()) * (1 + 1e-9) if not periodic else 1.0
    g = max(3, int(1.0 / (1.35 * math.sqrt(k / (math.pi * n)))))
    side = size / g
    cx = ((x - lo[0]) / side).long().clamp_(0, g - 1)
    cy = ((y - lo[1]) / side).long().clamp_(0, g - 1)
    cell = cx * g + cy
    order = torch.argsort(cell)
    count = torch.bincount(cell, minlength=g * g)
    start = torch.cumsum(count, 0) - count
    most = int(count.max())
    slot = torch.arange(most, device=x.device)
    parts = []
    for q in torch.split(every, max(1, (1 << 26) // (9 * most))):
        js, lives = [], []
        for a in (-1, 0, 1):
            for b in (-1, 0, 1):
                ex, ey = cx[q] + a, cy[q] + b
                inside = torch.ones_like(ex, dtype=torch.bool) if periodic else (ex >= 0) & (ex < g) & (ey >= 0) & (ey < g)
                c = (ex % g) * g + ey % g
                lives.append(inside[:, None] & (slot[None, :] < count[c][:, None]))
                js.append(order[(start[c][:, None] + slot[None, :]).clamp_(max=n - 1)])
        parts.append(pick(q[:, None], torch.cat(js, 1), torch.cat(lives, 1)))
    out = [torch.cat(t) for t in zip(*parts)]
    short = torch.nonzero(out[3][:, -1] > (side * (1 - 1e-6)) ** 2).flatten()  # the nine cells may miss some
    if short.numel():
        for t, b in zip(out, brute(short)):
            t[short] = b
    return out


def evaluate(p, x, y, vx, vy, u):
    j, rx, ry, d2 = nearest(x, y, p["k"], p["hor"], p["vert"])
    d = torch.sqrt(d2)
    h = d[:, -1]
    q = d / h[:, None]
    a = 1 - q
    if p["kernel"] == "Wendland":
        f, df = a ** 4 * (1 + 4 * q), -10 * q * a ** 3
        fp, dfp = 4 * 7 / (math.pi * 4), 8 * 7 / (math.pi * 4)
    else:
        low = q < 0.5
        f = torch.where(low, q ** 3 - q * q + 1 / 6, a ** 3 / 3)
        df = torch.where(low, 3 * q * q - 2 * q, -a * a)
        fp = dfp = 6 * 40 / (math.pi * 7)
    g, m = p["gamma"], p["mass"]
    rho = fp * m * f.sum(1) / h ** 2
    c = torch.sqrt(g * (g - 1) * u)
    ct = c * c / (g * rho)
    wx, wy = vx[j] - vx[:, None], vy[j] - vy[:, None]
    dot = wx * rx + wy * ry
    mean = lambda t: 0.5 * (t[:, None] + t[j])  # noqa: E731
    mu = dot * mean(h) / (rx * rx + ry * ry + p["etasq"])
    pi = torch.where(dot < 0, (-p["alpha"] * mean(c) * mu + p["beta"] * mu * mu) / mean(rho), torch.zeros_like(mu))
    w = (pi + ct[:, None] + ct[j]) * df / d
    s = m * dfp / h ** 3
    ax, ay = (rx * w).sum(1) * s + p["accel"][0], (ry * w).sum(1) * s + p["accel"][1]
    return ax, ay, ct * (dot * df).sum(1) * m, (rho, c, h), d


def restate(p, arrays, steps):
    """The state and derived fields after `steps` steps from an initial condition."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x, y, vx, vy, u = (torch.from_numpy(np.ascontiguousarray(a)).to(dev) for a in arrays)
    dth, derived = p["dth"], None
    ax, ay, udot, _, _ = evaluate(p, x, y, vx, vy, u)
    for _ in range(steps):
        x, y = x + vx * dth, y + vy * dth
        ax, ay, udot, derived, _ = evaluate(p, x, y, vx + ax * dth, vy + ay * dth, u + udot * dth)
        vx, vy, u = vx + ax * (2 * dth), vy + ay * (2 * dth), u + udot * 2 * dth
        x, y = x + vx * dth, y + vy * dth
        if p["hor"] != OPEN:  # at most one axis wraps per step
            (x0, x1), (y0, y1) = p["hor"], p["vert"]
            lx, hx = x < x0, x > x1
            ly, hy = ~lx & ~hx & (y < y0), ~lx & ~hx & (y > y1)
            x = torch.where(lx, x + (x1 - x0), torch.where(hx, x - (x1 - x0), x))
            y = torch.where(ly, y + (y1 - y0), torch.where(hy, y - (y1 - y0), y))
        l, r, t, b = p["refl"]
        vx = torch.where((x < l) | (x > r), -vx, vx)
        vy = torch.where((y < t) | (y > b), -vy, vy)
        x, y = x.clamp(l, r), y.clamp(t, b)
    return dict(zip(STATE + DERIVED, (x, y, vx, vy, u, ax, ay, udot) + derived))


def exact(case, seed):
    if sum(sizes(case)) > EXACT_MAX_N and case["kind"] != "ensemble":
        return None
    sims = inputs(case, seed)
    if case["kind"] == "noalloc":
        (p, arrays), = sims
        x, y = (torch.from_numpy(a) for a in arrays[:2])
        zero, one = torch.zeros_like(x), torch.ones_like(x)
        _, _, _, (rho, _, h), d = evaluate(p, x, y, zero, zero, one)
        return {"ids": None, "dist": d.flip(1).flatten(), "rho": rho, "h": h}
    got = [restate(p, a, PREP_STEPS + case["steps"]) for p, a in sims]
    out = {name: torch.cat([g[name] for g in got]) for name in STATE + DERIVED}
    if case["frame"]:
        out["rgba"] = None
    return out
