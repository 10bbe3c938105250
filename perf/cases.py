"""The workloads whose speed matters to users of fastlpr_b200, over the sizes
they come in: local polynomial fits in one to three dimensions (orders 0 to 2,
real, complex and several responses, full and learned bandwidth search, mean
and variance fits), many fits through one plan, and kernel density estimates.

``listed()`` gives the standing cases, ``draw(rng)`` one more of the same
ranges; ``prepare`` makes a case's inputs from a seed, ``run`` is one pass
through the public calls, ``work`` the bytes and operations it cannot do
without, and ``exact`` the same results in 64-bit torch.
"""
import math

import numpy as np
import torch

import fastlpr_b200

TAPS = 9          # spreading taps per axis at the default accuracy (n >= 100)
PROBES = 10       # Hutchinson probes of the degrees of freedom (the default)

# Every case has these keys; a missing one takes its value here.
DEFAULTS = {
    "kind": "lpr",        # lpr, device, pair, plan, kde
    "n": 1000, "d": 1, "order": 1,
    "g0": 0, "g1": 0, "g2": 0,            # grid per axis (0: the library's default grid)
    "H": 20, "hlo": 0.01, "hhi": 1.0, "Hb": 0,   # Hb > 0: an H x Hb list, its own bandwidth per axis
    "dy": 1, "complex": False, "search": "full",
    "new": 0,             # new points at which the fit is then evaluated
    "problems": 0,
    "kernel": "gaussian",
}


def _full(case):
    return {**DEFAULTS, **case}


def listed():
    return [
        # interactive use: a handful of points, everything at its default; launches and host work count
        {"name": "lpr1d_small", "kind": "lpr", "n": 800, "d": 1, "order": 1, "H": 20, "hlo": 0.05, "hhi": 1.0},
        # the ordinary 1-D curve fit of the benchmark's 1-D configuration
        {"name": "lpr1d_curve", "kind": "lpr", "n": 100000, "d": 1, "order": 1, "g0": 1024, "H": 20,
         "hlo": 0.01, "hhi": 1.0},
        # a complex-valued signal, local quadratic: the 64-bit grids in one dimension
        {"name": "lpr1d_quadratic_complex", "kind": "lpr", "n": 50021, "d": 1, "order": 2, "g0": 1024,
         "H": 24, "hlo": 0.005, "hhi": 0.5, "complex": True},
        # a small surface at the defaults: below 5000 points GCV and DoF go through the cubic spline
        {"name": "lpr2d_small_cubic", "kind": "lpr", "n": 3000, "d": 2, "order": 1, "H": 20, "hlo": 0.1,
         "hhi": 1.0},
        # two responses on a ragged grid, a bandwidth per axis, then prediction at new points
        {"name": "lpr2d_ragged_predict", "kind": "lpr", "n": 250007, "d": 2, "order": 0, "g0": 300, "g1": 421,
         "H": 5, "Hb": 5, "hlo": 0.02, "hhi": 0.5, "dy": 2, "new": 100003},
        # the benchmark's own fit, data already on the GPU
        {"name": "lpr2d_device", "kind": "device", "n": 1000000, "d": 2, "order": 1, "g0": 512, "g1": 512,
         "H": 32, "hlo": 0.005, "hhi": 0.5},
        # the same fit with the learned bandwidth search
        {"name": "lpr2d_device_learned", "kind": "device", "n": 1000000, "d": 2, "order": 1, "g0": 512,
         "g1": 512, "H": 32, "hlo": 0.005, "hhi": 0.5, "search": "learned"},
        # heteroscedastic regression: a local quadratic mean fit and the variance fit of the squared deviations
        {"name": "lpr2d_quadratic_pair", "kind": "pair", "n": 2000000, "d": 2, "order": 2, "g0": 512,
         "g1": 512, "H": 32, "hlo": 0.005, "hhi": 0.5},
        # a volume: local linear in three dimensions
        {"name": "lpr3d_volume", "kind": "lpr", "n": 100000, "d": 3, "order": 1, "g0": 64, "g1": 64, "g2": 64,
         "H": 8, "hlo": 0.05, "hhi": 0.5},
        # a day's batch of uneven data sets, new responses on known designs, through one plan
        {"name": "plan_uneven", "kind": "plan", "n": 50000, "problems": 12, "H": 24, "hlo": 0.005, "hhi": 0.5},
        # a density of two variables at the default grid
        {"name": "kde2d", "kind": "kde", "n": 30011, "d": 2, "H": 20, "hlo": 0.02, "hhi": 0.5},
        # the largest: the 3-D density of the benchmark configurations
        {"name": "kde3d_large", "kind": "kde", "n": 10000000, "d": 3, "g0": 128, "g1": 128, "g2": 128, "H": 16,
         "hlo": 0.01, "hhi": 0.3},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lpr1d", "lpr1d", "lpr2d", "lpr2d", "device", "learned", "pair", "lpr3d", "plan", "kde",
                       "kde", "kde3d"])
    hlo = round(rng.uniform(0.01, 0.1), 4)
    c = {"hlo": hlo, "hhi": round(hlo * rng.uniform(8.0, 40.0), 4)}
    if kind == "lpr1d":
        c |= {"kind": "lpr", "d": 1, "n": _log_int(rng, 500, 400000), "order": rng.choice([0, 1, 1, 2]),
              "H": rng.randint(8, 32), "g0": rng.choice([0, _log_int(rng, 100, 2048)]),
              "complex": rng.random() < 0.25, "new": rng.choice([0, _log_int(rng, 100, 100000)])}
        if c["n"] > 60000 and not c["g0"]:
            c["g0"] = 1024
    elif kind == "lpr2d":
        c |= {"kind": "lpr", "d": 2, "n": _log_int(rng, 1500, 1000000), "order": rng.choice([0, 1, 1, 2]),
              "H": rng.randint(6, 32), "g0": _log_int(rng, 48, 512), "g1": _log_int(rng, 48, 512),
              "dy": rng.choice([1, 1, 2]), "new": rng.choice([0, _log_int(rng, 100, 100000)])}
    elif kind in ("device", "learned"):
        c |= {"kind": "device", "d": 2, "n": _log_int(rng, 20000, 1200000), "order": rng.choice([0, 1]),
              "H": rng.randint(12, 32), "search": "learned" if kind == "learned" else "full"}
        c["g0"] = c["g1"] = _log_int(rng, 100, 512)
    elif kind == "pair":
        c |= {"kind": "pair", "d": 2, "n": _log_int(rng, 50000, 1500000), "order": 2, "H": rng.randint(8, 24),
              "g0": _log_int(rng, 100, 512), "g1": _log_int(rng, 100, 512)}
    elif kind == "lpr3d":
        c |= {"kind": "lpr", "d": 3, "n": _log_int(rng, 6000, 200000), "order": rng.choice([0, 1]),
              "H": rng.randint(4, 8), "g0": rng.randint(24, 64), "g1": rng.randint(24, 64),
              "g2": rng.randint(24, 64)}
        c["hlo"] = max(c["hlo"], 0.05)
    elif kind == "plan":
        c |= {"kind": "plan", "n": _log_int(rng, 5000, 50000), "problems": rng.randint(4, 12),
              "H": rng.randint(12, 24)}
    elif kind == "kde":
        c |= {"kind": "kde", "d": rng.choice([1, 2]), "n": _log_int(rng, 500, 1000000), "H": rng.randint(8, 32),
              "kernel": rng.choice(["gaussian", "gaussian", "epanechnikov"])}
        c["g0"] = _log_int(rng, 60, 512)
        c["g1"] = _log_int(rng, 60, 512)
    else:
        c |= {"kind": "kde", "d": 3, "n": _log_int(rng, 20000, 6000000), "H": rng.randint(4, 16)}
        c["g0"] = c["g1"] = c["g2"] = rng.randint(32, 128)
        c["hlo"] = max(c["hlo"], 0.03)
        c["hhi"] = max(c["hhi"], 3 * c["hlo"])
    return c


# --------------------------------------------------------------------------
# Inputs
# --------------------------------------------------------------------------
def _grid(c):
    if c["g0"]:
        return [c["g0"], c["g1"], c["g2"]][:c["d"]]
    g = int(math.ceil(c["n"] ** (1.0 / c["d"])))
    return [g] * c["d"]


def _bandwidths(c):
    if c["Hb"]:
        return fastlpr_b200.get_hlist([c["H"], c["Hb"]], np.array([[c["hlo"], c["hhi"]]] * 2))
    hv = np.logspace(math.log10(c["hlo"]), math.log10(c["hhi"]), c["H"])
    return np.column_stack([hv] * c["d"])


def _points(c, g):
    """Points on the GPU: uniform for regression, a mixture of eight normals with a uniform tenth for densities."""
    n, d, dev = c["n"], c["d"], "cuda"
    if c["kind"] != "kde":
        return torch.rand((n, d), generator=g, device=dev, dtype=torch.float64)
    mean = 0.2 + 0.6 * torch.rand((8, d), generator=g, device=dev, dtype=torch.float64)
    sd = 0.02 + 0.08 * torch.rand((8, d), generator=g, device=dev, dtype=torch.float64)
    comp = torch.randint(0, 8, (n,), generator=g, device=dev)
    x = mean[comp] + sd[comp] * torch.randn((n, d), generator=g, device=dev, dtype=torch.float64)
    back = torch.rand(n, generator=g, device=dev) < 0.1
    u = torch.rand((n, d), generator=g, device=dev, dtype=torch.float64)
    return torch.where(back[:, None], u, x)


def _response(c, x, g):
    n = x.shape[0]

    def noise():
        return torch.randn(n, generator=g, device=x.device, dtype=torch.float64)

    f = torch.sin(2 * math.pi * x[:, 0])
    if c["d"] > 1:
        f = f * torch.cos(2 * math.pi * x[:, 1])
    if c["d"] > 2:
        f = f + x[:, 2]
    if c["complex"]:
        return torch.complex(torch.cos(2 * math.pi * x[:, 0]) + 0.1 * noise(), f + 0.1 * noise())
    if c["dy"] > 1:
        return torch.stack([(1 + k) * f + 0.1 * noise() for k in range(c["dy"])], dim=1)
    return f + 0.1 * noise()


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _plan_cases(c):
    """The uneven problems of a plan (their sizes go with the case, not with the seed): half of them curves on
    1024 grid points, half surfaces on 256 x 256, sizes lognormal about n, a quarter of them complex."""
    rng = np.random.default_rng(7)
    out = []
    for k in range(c["problems"]):
        n = int(np.clip(round(c["n"] * math.exp(rng.standard_normal())), 1000, 1000000))
        d = 1 if k % 2 == 0 else 2
        out.append({**c, "kind": "lpr", "n": n, "d": d, "order": int(rng.integers(0, 3)),
                    "g0": 1024 if d == 1 else 256, "g1": 256, "complex": k % 4 == 3})
    return out


def _options(c):
    o = {"order": c["order"]}
    if c["g0"]:
        o["N"] = _grid(c)
    if c["search"] != "full":
        o["bandwidth_search"] = c["search"]
    return o


def _inputs(c, seed):
    """The case's arrays on the GPU; prepare() and exact() start from the same ones."""
    g = _generator(seed)
    x = _points(c, g)
    if c["kind"] == "kde":
        return {"x": x}
    if c["kind"] == "pair":
        sigma = 0.05 + 0.1 * x[:, 0]
        e = sigma * torch.randn(c["n"], generator=g, device=x.device, dtype=torch.float64)
        return {"x": x, "y": torch.sin(2 * math.pi * x[:, 0]) * torch.cos(2 * math.pi * x[:, 1]) + e, "v": e * e}
    new = torch.rand((c["new"], c["d"]), generator=g, device=x.device, dtype=torch.float64)
    return {"x": x, "y": _response(c, x, g), "new": new}


def prepare(case, seed):
    c = _full(case)
    if c["kind"] == "plan":
        probs = []
        for k, p in enumerate(_plan_cases(c)):
            a = _inputs(p, int(seed) * 1009 + k)
            probs.append((a["x"].cpu().numpy(), a["y"].cpu().numpy(), _bandwidths(p), _options(p)))
        return {"case": c, "plan": fastlpr_b200.LprPlan(probs), "ys": [p[1] for p in probs]}
    a = _inputs(c, seed)
    if c["kind"] != "device":
        a = {k: v.cpu().numpy() for k, v in a.items()}
    o = _options(c)
    if c["kind"] == "kde":
        o = {"kernel_type": c["kernel"]}
        if c["g0"]:
            o["N"] = _grid(c)
    return {"case": c, "h": _bandwidths(c), "options": o, **a}


# --------------------------------------------------------------------------
# One pass
# --------------------------------------------------------------------------
def _fit_outputs(r):
    g = r.gcv_yhat
    out = {"yhat": r.yhat, "residuals": r.metadata["residuals"], "surface": r.fpp_yhat.values, "s0": r.s0,
           "gcv": g["gcv_m"], "gcv_sd": g["gcv_sd"], "dof": g["dof"], "dof_stderr": g["dof_stderr"],
           "h": r.h, "choice": int(g["id1se"])}
    if r.d is not None:
        out["d"] = r.d
    return out


def run(state):
    c = state["case"]
    if c["kind"] == "plan":
        regs = state["plan"].run(state["ys"])
        return {"fits": [{"yhat": r.yhat, "residuals": r.metadata["residuals"], "surface": r.fpp_yhat.values,
                          "s0": r.s0} for r in regs],
                "scores": np.stack([[r.gcv_yhat[k] for k in ("gcv_m", "gcv_sd", "dof", "dof_stderr")]
                                    for r in regs]),
                "choice": np.array([r.gcv_yhat["id1se"] for r in regs])}
    if c["kind"] == "kde":
        k = fastlpr_b200.cv_fastkde(state["x"], state["h"], state["options"])
        return {"fhat": k.fhat, "all": k.metadata["fhat_all"], "lcv": k.lcv["lcv_m"], "lcv_sd": k.lcv["lcv_sd"],
                "h": k.h, "choice": int(k.lcv["id1se"])}
    if c["kind"] == "device":
        return _fit_outputs(fastlpr_b200.cv_fastlpr_device(state["x"], state["y"], state["h"], state["options"]))
    r = fastlpr_b200.cv_fastlpr(state["x"], state["y"], state["h"], state["options"])
    out = _fit_outputs(r)
    if c["kind"] == "pair":
        v = fastlpr_b200.cv_fastlpr(state["x"], state["v"], state["h"], {**state["options"], "y_type_out": "variance"})
        return {"mean": out, "variance": _fit_outputs(v)}
    if c["new"]:
        out["predicted"] = fastlpr_b200.fastlpr_predict(r, state["new"])
    return out


# --------------------------------------------------------------------------
# What a pass cannot do without
# --------------------------------------------------------------------------
def _padded(G):
    return [2 ** int(math.ceil(math.log2(2 * g - 1))) for g in G]


def _terms(d, order):
    return math.comb(d + order, order)


def _fit_work(c):
    n, d, G = c["n"], c["d"], _grid(c)
    M, L = math.prod(G), math.prod(_padded(G))
    H = c["H"] * max(1, c["Hb"]) if c["search"] == "full" else 5
    ny = c["dy"] * (2 if c["complex"] else 1)
    nt = _terms(d, c["order"])
    ns = len({tuple(a + b for a, b in zip(p, q)) for p in _powers(d, c["order"]) for q in _powers(d, c["order"])})
    fft = 2.5 * L * math.log2(L)          # a real transform of the padded grid
    flops = 2.0 * n * (1 + ny + PROBES) * TAPS ** d + (1 + ny + PROBES) * fft
    flops += H * (ns + nt * (ny + PROBES)) * (fft + 6.0 * L / 2) + H * M * (nt ** 3 / 3.0 + 2.0 * nt * (ny + PROBES))
    # points, responses and probes read; fitted values, residuals, the surface and s0 written
    data = 8.0 * (n * (d + ny + PROBES) + 2 * n * ny + M * (ny + 1) + c["new"] * (d + ny))
    return data, flops


def work(case):
    c = _full(case)
    if c["kind"] == "plan":
        parts = [_fit_work(p) for p in _plan_cases(c)]
        # the designs are the plan's
        return {"bytes": sum(b - 8.0 * p["n"] * (p["d"] + PROBES) for (b, _), p in zip(parts, _plan_cases(c))),
                "flops": sum(f for _, f in parts)}
    if c["kind"] == "kde":
        G = _grid(c)
        M, L = math.prod(G), math.prod(_padded(G))
        fft = 2.5 * L * math.log2(L)
        return {"bytes": 8.0 * (c["n"] * c["d"] + M * c["H"]),
                "flops": 2.0 * c["n"] * TAPS ** c["d"] + (1 + c["H"]) * fft
                + c["H"] * (3.0 * L + c["n"] * (2.0 * 2 ** c["d"] + 20))}
    data, flops = _fit_work(c)
    return {"bytes": data * (2 if c["kind"] == "pair" else 1), "flops": flops * (2 if c["kind"] == "pair" else 1)}


# --------------------------------------------------------------------------
# The same results in 64 bits: the estimators' definition, in torch
# --------------------------------------------------------------------------
def _powers(d, order):
    out = []
    for total in range(order + 1):
        if d == 1:
            out.append((total,))
        elif d == 2:
            out += [(p, total - p) for p in range(total, -1, -1)]
        else:
            out += [(p, q, total - p - q) for p in range(total, -1, -1) for q in range(total - p, -1, -1)]
    return out


class _Grid:
    """Scaled data, padded grid and knots of one data set (mean 0, ddof-1 deviation 1, mid-range at 0)."""

    def __init__(self, x, G):
        n, d = x.shape
        self.x, self.n, self.d, self.G, self.L = x, n, d, G, _padded(G)
        self.mean, self.std = x.mean(0), x.std(0)
        self.xmin, self.xmax = x.amin(0), x.amax(0)
        lo, hi = (self.xmin - self.mean) / self.std, (self.xmax - self.mean) / self.std
        center = (lo + hi) / 2
        self.lo, self.hi = lo - center, hi - center
        xs = (x - self.mean) / self.std - center
        self.axes = [torch.linspace(float(self.lo[a]), float(self.hi[a]), G[a], dtype=torch.float64, device=x.device)
                     for a in range(d)]
        self.crop = [-(-(L - g) // 2) for L, g in zip(self.L, G)]
        self.knots = []
        for a in range(d):
            L, g = self.L[a], G[a]
            q = (L - g) // 2
            idx = np.linspace(-0.5, 0.5 - 1 / L, L)
            span, first = idx[q + g - 1] - idx[q], idx[q]

            def place(v):
                return torch.remainder((v - self.lo[a]) / (self.hi[a] - self.lo[a]) * span + first + 0.5, 1.0) - 0.5

            shift = -0.5 - ((place(self.lo[a]) + place(self.hi[a])) * 0.5 - 0.5)
            self.knots.append(torch.remainder((place(xs[:, a]) + shift) * (2 * math.pi), 2 * math.pi))

    def spectra(self, channels):
        """Gaussian gridding of (C, n) channels with 9 taps per axis, transformed and divided by n."""
        dev, n, C = self.x.device, self.n, channels.shape[0]
        first, weights, cells = [], [], []
        for a, k in enumerate(self.knots):
            L = self.L[a]
            hx, tau = 2 * math.pi / L, math.pi * 4 / (L * L * 0.5)
            m = torch.round(k / hx)
            taps = torch.arange(-4, 5, device=dev)
            diff = k[:, None] - hx * (m[:, None] + taps)
            weights.append(torch.exp(-diff * diff / (4 * tau)))
            cells.append(torch.remainder(m.long()[:, None] + taps, L))
        out = torch.zeros((C, math.prod(self.L)), dtype=torch.float64, device=dev)
        for combo in np.ndindex(*([TAPS] * self.d)):
            w = torch.ones(n, dtype=torch.float64, device=dev)
            cell = torch.zeros(n, dtype=torch.int64, device=dev)
            for a, j in enumerate(combo):
                w = w * weights[a][:, j]
                cell = cell * self.L[a] + cells[a][:, j]
            for k in range(C):
                out[k].index_add_(0, cell, channels[k] * w)
        dims = tuple(range(1, self.d + 1))
        return torch.fft.rfftn(out.reshape([C] + self.L), dim=dims) / n

    def _pad(self, a, values):
        full = torch.zeros(values.shape[:-1] + (self.L[a],), dtype=torch.float64, device=self.x.device)
        at = (self.L[a] - self.G[a]) // 2 + 1
        full[..., at:at + self.G[a]] = values
        return full

    def kernel(self, h, powers, name):
        """Half spectrum of K(u) u^powers / prod h on the padded grid for one bandwidth row."""
        if name == "gaussian":
            k = None
            for a in range(self.d):
                u = self.axes[a] / h[a]
                f = self._pad(a, torch.exp(-0.5 * u * u) * u ** powers[a] / h[a])
                f = torch.fft.rfft(f) if a == self.d - 1 else torch.fft.fft(f)
                k = f if k is None else k[..., None] * f
            return k / math.sqrt(2 * math.pi)
        mesh = torch.meshgrid(*[ax / float(v) for ax, v in zip(self.axes, h)], indexing="ij")
        ssq = sum(u * u for u in mesh)
        k = torch.clamp(0.75 * (1 - ssq), min=float(np.finfo(float).eps)) / float(np.prod(h))
        for u, p in zip(mesh, powers):
            k = k * u ** p
        full = torch.zeros(self.L, dtype=torch.float64, device=self.x.device)
        at = tuple(slice((L - g) // 2 + 1, (L - g) // 2 + 1 + g) for L, g in zip(self.L, self.G))
        full[at] = k
        return torch.fft.rfftn(full)

    def convolve(self, spectra, kernel):
        dims = tuple(range(1, self.d + 1))
        full = torch.fft.irfftn(spectra * kernel, s=self.L, dim=dims)
        sl = (slice(None),) + tuple(slice(q, q + g) for q, g in zip(self.crop, self.G))
        return full[sl].reshape(spectra.shape[0], -1)


def _interpolate(lo, hi, G, values, pts):
    """Clamped multilinear interpolation of (C, M) grid values at pts."""
    n, d = pts.shape
    ix, fr = [], []
    for a in range(d):
        ax = np.linspace(float(lo[a]), float(hi[a]), G[a])
        t = (pts[:, a] - ax[0]) / (ax[1] - ax[0])
        i = t.floor().clamp(0, G[a] - 2)
        ix.append(i.long())
        fr.append((t - i).clamp(0.0, 1.0))
    out = torch.zeros((values.shape[0], n), dtype=torch.float64, device=pts.device)
    for corner in np.ndindex(*([2] * d)):
        w = torch.ones(n, dtype=torch.float64, device=pts.device)
        at = torch.zeros(n, dtype=torch.int64, device=pts.device)
        for a, b in enumerate(corner):
            w = w * (fr[a] if b else 1.0 - fr[a])
            at = at * G[a] + ix[a] + b
        out += w * values[:, at]
    return out


def _spline_basis(axis, x):
    """(len(x), len(axis)) values of the not-a-knot cubic B-splines on the axis, end pieces extended."""
    t = np.concatenate([[axis[0]] * 4, axis[2:-2], [axis[-1]] * 4])
    last = len(t) - 5
    span = np.clip(np.searchsorted(t, x, side="right") - 1, 3, last)
    b = np.zeros((len(x), len(t) - 1))
    b[np.arange(len(x)), span] = 1.0
    for k in range(1, 4):
        nxt = np.zeros((len(x), len(t) - 1 - k))
        for i in range(len(t) - 1 - k):
            if t[i + k] > t[i]:
                nxt[:, i] += (x - t[i]) / (t[i + k] - t[i]) * b[:, i]
            if t[i + k + 1] > t[i + 1]:
                nxt[:, i] += (t[i + k + 1] - x) / (t[i + k + 1] - t[i + 1]) * b[:, i + 1]
        b = nxt
    return b


def _spline_interpolator(lo, hi, G, pts):
    """A function of (C, M) grid values: their not-a-knot cubic spline at pts."""
    host, maps = pts.cpu().numpy(), []
    for a in range(len(G)):
        ax = np.linspace(float(lo[a]), float(hi[a]), G[a])
        at = np.linalg.solve(_spline_basis(ax, ax).T, _spline_basis(ax, host[:, a]).T).T
        maps.append(torch.from_numpy(np.ascontiguousarray(at)).to(pts.device))

    def evaluate(values):
        v = values.reshape([values.shape[0]] + list(G))
        v = torch.einsum("cg...,ng->cn...", v, maps[0])
        for m in maps[1:]:
            v = torch.einsum("cng...,ng->cn...", v, m)
        return v

    return evaluate


def _exact_fit(c, x, y, new, variance=False):
    dev, n, d, order, G = x.device, c["n"], c["d"], c["order"], _grid(c)
    grid = _Grid(x, G)
    raw = y
    if variance:
        y = torch.log(y + 1.0 / n)
    cols = torch.stack([y.real, y.imag]) if c["complex"] else (y.t() if y.dim() == 2 else y[None])
    ny = cols.shape[0]
    probes = torch.from_numpy(np.random.Generator(np.random.MT19937(42)).standard_normal((n, PROBES))).to(dev).t()
    spec = grid.spectra(torch.cat([torch.ones((1, n), dtype=torch.float64, device=dev), cols, probes]))
    hs = _bandwidths(c)
    H, M, pw = len(hs), math.prod(G), _powers(d, order)
    nt = len(pw)
    S = torch.empty((H, nt, nt, M), dtype=torch.float64, device=dev)
    for k, h in enumerate(hs):
        done = {}
        for i in range(nt):
            for j in range(i + 1):
                e = tuple(p + q for p, q in zip(pw[i], pw[j]))
                if e not in done:
                    done[e] = grid.convolve(spec[:1], grid.kernel(h, e, "gaussian"))[0]
                S[k, i, j] = S[k, j, i] = done[e]
    if order == 0:
        S = S + float(np.finfo(float).eps)
        level = float(S.max()) * 1e-8
    else:
        level = 1e-6 * max(float(S[:, i, i].abs().max()) for i in range(nt))
    cubic = d > 1 and n < 5000
    at = _spline_interpolator(grid.xmin, grid.xmax, G, x) if cubic else (
        lambda v: _interpolate(grid.xmin, grid.xmax, G, v, x))
    pp = (probes * probes).sum(1)
    gcv, sd, dof, dof_se, keep = [], [], [], [], []
    for k, h in enumerate(hs):
        if order == 0:
            m = grid.convolve(spec[1:], grid.kernel(h, pw[0], "gaussian")) / torch.clamp(S[k, 0, 0], min=level)
        else:
            A = S[k].permute(2, 0, 1) + level * torch.eye(nt, dtype=torch.float64, device=dev)
            e1 = torch.zeros((M, nt, 1), dtype=torch.float64, device=dev)
            e1[:, 0] = 1.0
            z = torch.linalg.solve(A, e1)[..., 0]
            m = sum(z[:, i] * grid.convolve(spec[1:], grid.kernel(h, pw[i], "gaussian")) for i in range(nt))
        fit = at(m)
        tr = (n * (fit[ny:] * probes).sum(1) / pp).clamp(0.0, float(n))
        rest = 1 - tr / n
        if c["complex"]:
            rest = 2 * rest - 1
        rest = rest.clamp(0.0, 1.0)
        pen = 1.0 / rest.clamp(min=0.01) ** 2
        rss = ((cols - fit[:ny]) ** 2).sum(1)
        mse = float((rss.sum() if c["complex"] else rss[0]) / n)
        gcv.append(mse * float(pen.mean()))
        sd.append(mse * float(pen.std()))
        dof.append(n * (1 - float(rest.mean())) if c["complex"] else float(tr.mean()))
        dof_se.append(float(tr.std()) / math.sqrt(PROBES))
        keep.append(m[:ny])
    b = int(np.argmin(gcv))
    surface = keep[b]
    yhat = _interpolate(grid.xmin, grid.xmax, G, surface, x)
    out = {"s0": S[b, 0, 0].reshape(G), "gcv": np.array(gcv), "gcv_sd": np.array(sd), "dof": np.array(dof),
           "dof_stderr": np.array(dof_se), "h": hs[b], "choice": b}
    if variance:
        out["d"] = 1.0 / float((raw * torch.exp(-yhat[0])).mean())
        yhat, surface = torch.exp(yhat) / out["d"], torch.exp(surface) / out["d"]

    def shape(v, lead):
        if c["complex"]:
            return torch.complex(v[0], v[1]).reshape(lead)
        return v[0].reshape(lead) if ny == 1 else v.t().reshape(lead + [ny])

    out["yhat"], out["surface"] = shape(yhat, [n]), shape(surface, list(G))
    out["residuals"] = raw - out["yhat"]
    if c["new"]:
        out["predicted"] = shape(_interpolate(grid.xmin, grid.xmax, G, surface, new), [c["new"]])
    return {k: v.cpu().numpy() if torch.is_tensor(v) else v for k, v in out.items()}


def _exact_kde(c, x):
    n, d, G = c["n"], c["d"], _grid(c)
    grid = _Grid(x, G)
    spec = grid.spectra(torch.ones((1, n), dtype=torch.float64, device=x.device))
    hs = _bandwidths(c)
    cell = float(np.prod([float(grid.std[a] * (grid.hi[a] - grid.lo[a])) / (G[a] - 1) for a in range(d)]))
    fs, lcv, sd = [], [], []
    for h in hs:
        s = grid.convolve(spec, grid.kernel(h, (0,) * d, c["kernel"])) + float(np.finfo(float).eps)
        f = (s / (s.sum() * cell)).clamp(min=0.0)
        at = _interpolate(grid.xmin, grid.xmax, G, f, x)[0]
        k0 = 1.0 / math.sqrt(2 * math.pi) / float(np.prod(h))
        lg = torch.log(torch.clamp(n / (n - 1) * (at - k0 / n), min=1e-10))
        fs.append(f[0].reshape(G))
        lcv.append(float(lg.sum()))
        sd.append(float(lg.std(correction=0)) * math.sqrt(n))
    b = int(np.argmax(lcv))
    near = [i for i in range(len(hs)) if lcv[i] >= lcv[b] - sd[b]]
    pick = near[int(np.argmax([hs[i].sum() for i in near]))]
    return {"fhat": fs[pick].cpu().numpy(), "all": torch.stack(fs, -1).cpu().numpy(), "lcv": np.array(lcv),
            "lcv_sd": np.array(sd), "h": hs[pick], "choice": pick}


def exact(case, seed):
    c = _full(case)
    if c["search"] != "full" or c["n"] * TAPS ** c["d"] > 8e9:
        return None       # a learned window is the network's choice; larger 3-D griddings take too long
    if c["kind"] == "plan":
        fits = []
        for k, p in enumerate(_plan_cases(c)):
            a = _inputs(p, int(seed) * 1009 + k)
            fits.append(_exact_fit(p, a["x"], a["y"], None))
        return {"fits": [{k: f[k] for k in ("yhat", "residuals", "surface", "s0")} for f in fits],
                "scores": np.stack([[f[k] for k in ("gcv", "gcv_sd", "dof", "dof_stderr")] for f in fits]),
                "choice": np.array([f["choice"] for f in fits])}
    a = _inputs(c, seed)
    if c["kind"] == "kde":
        return _exact_kde(c, a["x"])
    mean = _exact_fit(c, a["x"], a["y"], a.get("new"))
    if c["kind"] == "pair":
        return {"mean": mean, "variance": _exact_fit(c, a["x"], a["v"], None, variance=True)}
    return mean
