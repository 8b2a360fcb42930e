"""What the framework is timed on: its public entry points over the range of networks, boxes and
options that its users run.

A case is a dict of plain values.  `kind` says which entry point one pass calls:
  action     FSPMat.action           y += A(t) x, the operator by itself
  transpose  FSPMat.apply_transpose  y = A^T x, the operator of the adjoint solves
  expv       KryExpvFSP.solve        exp(tA) p, a new solver for each solve as callers make it
  bdf        BDFIntegrator           time-varying rates, from t = 0 to one output time
  batch      BatchKrylov.solve       exp(tA_i) p_i for many parameter sets of one network
  gradient   Likelihood.gradient     log L and its gradient in all rates
`net` names a network of cuda_fsp_b200.models and `box` its largest counts, species 0 first.  The seed
draws the rates (around the network's own), the vectors, the start distributions and the data.
All values are 64-bit.
"""
import math

import numpy as np
import torch

from cuda_fsp_b200 import BatchKrylov, BDFIntegrator, FSPMat, KryExpvFSP, Likelihood, MatrixFormat, models

FORMATS = {"kron": MatrixFormat.KRONECKER, "csr": MatrixFormat.CUDA_CSR, "hyb": MatrixFormat.HYB}


def listed():
    return [
        # One operator call on a small toggle switch with time-varying rates, as an external integrator
        # calls it thousands of times: launch and host latency.  Both box sides are odd in states.
        {"name": "action toggle 101x81", "kind": "action", "net": "toggle", "box": "100x80", "format": "kron"},
        # The operator on the 3-species mass-action network at 16.8M states, the headline size.
        {"name": "action mass3 255^3", "kind": "action", "net": "mass3", "box": "255x255x255", "format": "kron"},
        # The operator on the 12-reaction gene network: five species, binary genes, two long mRNA axes.
        {"name": "action gene 8M", "kind": "action", "net": "gene", "box": "1x1x1x127x8191", "format": "kron"},
        # The sparse format (propensities that need not factorise), a box with unequal ragged sides.
        {"name": "action mass3 csr 3M", "kind": "action", "net": "mass3", "box": "159x150x131", "format": "csr"},
        # The transposed operator (backward direction) on a ragged 3-species box.
        {"name": "transpose mass3 4M", "kind": "transpose", "net": "mass3", "box": "210x149x127"},
        # The smallest solve: two species, 32,768 states, m = 30 with full orthogonalisation.
        {"name": "expv birth-death 32K", "kind": "expv", "net": "birth_death", "box": "127x255", "t": 10.0, "m": 30, "q": 0,
         "tol": 1e-9},
        # An ordinary solve: the gene network on an uneven box.
        {"name": "expv gene 134K", "kind": "expv", "net": "gene", "box": "1x1x1x110x150", "t": 5.0, "m": 30, "q": 0, "tol": 1e-9},
        # A large stiff solve with full orthogonalisation (the default), over a short horizon.
        {"name": "expv mass3 255^3 full", "kind": "expv", "net": "mass3", "box": "255x255x255", "t": 0.012, "m": 30, "q": 0,
         "tol": 1e-8},
        # A large stiff solve with the options that serve such networks best: m = 60, incomplete
        # orthogonalisation against 3 vectors; ragged box.
        {"name": "expv mass3 5.5M iop", "kind": "expv", "net": "mass3", "box": "191x179x160", "t": 0.05, "m": 60, "q": 3,
         "tol": 1e-8},
        # The time-varying gene model from its start through the switch of its first gene at t = 5.
        {"name": "bdf gene 131K", "kind": "bdf", "net": "gene", "box": "1x1x1x127x127", "t": 6.0, "rtol": 1e-8, "atol": 1e-14},
        # A parameter sweep: many gene models with uneven boxes in one launch.
        {"name": "batch gene 48", "kind": "batch", "net": "gene", "sets": 48, "lo": 40, "hi": 120, "t": 2.0, "m": 30, "tol": 1e-9,
         "cluster": 8, "threads": 512},
        # One gradient of the log-likelihood of single-cell counts, as an optimiser asks for it; the
        # tolerance is one that keeps rarely visited cells exact.
        {"name": "gradient gene 131K", "kind": "gradient", "net": "gene", "box": "1x1x1x127x127", "t": 16.0, "times": 4,
         "m": 30, "tol": 1e-12},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(*b):
    return "x".join(str(int(v)) for v in b)


def draw(rng):
    kind = rng.choice(["action", "action", "transpose", "expv", "expv", "expv", "bdf", "batch", "gradient"])
    if kind in ("action", "transpose"):
        net = rng.choice(["toggle", "mass3", "gene"])
        fmt = rng.choice(["kron", "kron", "csr", "hyb"]) if kind == "action" else "kron"
        if net == "toggle":
            box = _box(_log_int(rng, 30, 2000), _log_int(rng, 30, 2000))
        elif net == "mass3":
            top = 150 if fmt != "kron" else 240
            box = _box(*(_log_int(rng, 24, top) for _ in range(3)))
        else:
            box = _box(1, 1, 1, _log_int(rng, 40, 200), _log_int(rng, 100, 3000 if fmt == "kron" else 1000))
        c = {"kind": kind, "net": net, "box": box}
        if kind == "action":
            c["format"] = fmt
        return c
    if kind == "expv":
        net = rng.choice(["birth_death", "gene", "mass3"])
        q = rng.choice([0, 0, 2, 3])
        m = rng.choice([20, 30, 30, 40]) if q == 0 else rng.choice([30, 45, 60])
        if net == "birth_death":
            box, t = _box(_log_int(rng, 60, 300), _log_int(rng, 100, 500)), round(rng.uniform(2.0, 10.0), 2)
        elif net == "gene":
            box, t = _box(1, 1, 1, _log_int(rng, 50, 160), _log_int(rng, 60, 300)), round(rng.uniform(1.0, 5.0), 2)
        else:
            box, t = _box(*(_log_int(rng, 50, 200) for _ in range(3))), round(rng.uniform(0.005, 0.03), 4)
        return {"kind": kind, "net": net, "box": box, "t": t, "m": m, "q": q, "tol": 1e-8 if net == "mass3" else 1e-9}
    if kind == "bdf":
        return {"kind": kind, "net": "gene", "box": _box(1, 1, 1, _log_int(rng, 50, 140), _log_int(rng, 50, 200)),
                "t": round(rng.uniform(1.0, 6.0), 2), "rtol": rng.choice([1e-6, 1e-8]), "atol": 1e-14}
    if kind == "batch":
        lo = _log_int(rng, 20, 60)
        return {"kind": kind, "net": "gene", "sets": _log_int(rng, 12, 64), "lo": lo, "hi": lo + _log_int(rng, 10, 60),
                "t": round(rng.uniform(0.5, 2.0), 2), "m": rng.choice([20, 30]), "tol": 1e-9, "cluster": rng.choice([4, 8]),
                "threads": rng.choice([256, 512])}
    return {"kind": "gradient", "net": "gene", "box": _box(1, 1, 1, _log_int(rng, 50, 127), _log_int(rng, 60, 127)),
            "t": round(rng.uniform(3.0, 16.0), 2), "times": rng.randint(2, 5), "m": 30, "tol": 1e-12}


# ---- inputs ----------------------------------------------------------------------------------------

def _bounds(case):
    return tuple(int(v) for v in case["box"].split("x"))


def _rng(seed):
    return np.random.default_rng(int(seed))


def _scale(rng, nr):
    return np.exp(rng.uniform(-0.25, 0.25, size=nr))


def _model(case, seed):
    rng, net = _rng(seed), case["net"]
    if net == "gene":
        return models.gene_expression(_bounds(case), time_varying=case["kind"] in ("action", "bdf"), rates_scale=_scale(rng, 12))
    if net == "toggle":
        return models.toggle(_bounds(case), time_varying=case["kind"] == "action")
    if net == "mass3":
        m = models.mass_action_3(bounds=_bounds(case))
    else:
        m = models.mass_action(_bounds(case), [[1, 0], [-1, 0], [0, 1], [0, -1]], [[0, 0], [1, 0], [1, 0], [0, 1]],
                               [10.0, 1.0, 0.5, 0.2], name="birth_death_2")
    m.rates = m.rates * _scale(rng, m.nr)
    return m


def _vectors(case, seed, n):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    x = torch.rand(n, generator=g, dtype=torch.float64, device="cuda")
    y = torch.rand(n, generator=g, dtype=torch.float64, device="cuda")
    return x / x.sum(), y / n


def _start(case, seed, bounds):
    """A start distribution: independent Poisson counts of the mRNA or species (genes off)."""
    rng = _rng(seed + 7)
    p = torch.ones(1, dtype=torch.float64, device="cuda")
    for b in bounds:
        k = torch.arange(b + 1, dtype=torch.float64, device="cuda")
        mean = rng.uniform(3.0, 7.0)
        f = torch.exp(k * math.log(mean) - mean - torch.lgamma(k + 1.0)) if b > 1 else torch.tensor(
            [1.0, 0.0], dtype=torch.float64, device="cuda")[:b + 1]
        p = torch.outer(f, p).reshape(-1)
    return p / p.sum()


def _times(case):
    return np.linspace(case["t"] / case["times"], case["t"], case["times"])


def _counts(case, seed, bounds):
    """Histograms of 1,000 cells per time over (nuclear, cytoplasmic) mRNA: over-dispersed counts around
    the gene model's mean course."""
    rng = _rng(seed + 13)
    nn, nc = bounds[3] + 1, bounds[4] + 1
    out = np.zeros((case["times"], nn * nc))
    for i, t in enumerate(_times(case)):
        mean_n = 1.5 * (1.0 - math.exp(-0.6 * t))
        mean_c = 15.0 * (1.0 - math.exp(-0.05 * t))
        shape = 0.5
        xn = np.minimum(rng.poisson(rng.gamma(shape, mean_n / shape, 1000)), 12)
        xc = np.minimum(rng.poisson(rng.gamma(shape, mean_c / shape, 1000)), 25)
        np.add.at(out[i], xn + nn * xc, 1.0)
    return out


def _batch_models(case, seed):
    rng = _rng(seed)
    shapes = _rng(case["sets"] * 1000 + case["lo"])  # the boxes belong to the sweep, the rates to the seed
    out = []
    for _ in range(case["sets"]):
        bn, bc = (int(v) for v in shapes.integers(case["lo"], case["hi"] + 1, size=2))
        out.append(models.gene_expression((1, 1, 1, bn, bc), time_varying=False,
                                          rates_scale=10.0 ** rng.uniform(-0.5, 0.5, size=12)))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        ms = _batch_models(case, seed)
        B = BatchKrylov.from_models(ms, m=case["m"], tol=case["tol"])
        B.set_shape(case["cluster"], case["threads"])
        p0 = torch.zeros(B.total, dtype=torch.float64, device="cuda")
        for i, m in enumerate(ms):
            p0[int(B.offsets[i]):int(B.offsets[i]) + m.n_states] = _start(case, seed + i, m.bounds)
        return {"kind": kind, "B": B, "t": case["t"], "p0": p0, "p": torch.empty_like(p0)}
    m = _model(case, seed)
    if kind == "gradient":
        return {"kind": kind, "L": Likelihood(m, _times(case), _counts(case, seed, m.bounds), n_marginal=3, kry_tol=case["tol"],
                                              m=case["m"]), "c": m.coefs(0.0)}
    A = FSPMat.from_model(m, FORMATS[case.get("format", "kron")])
    if kind in ("action", "transpose"):
        x, y = _vectors(case, seed, m.n_states)
        return {"kind": kind, "A": A, "x": x, "y": y, "c": m.coefs(0.0), "t": 1.0}
    p0 = _start(case, seed, m.bounds)
    s = {"kind": kind, "A": A, "p0": p0, "p": torch.empty_like(p0), "t": case["t"]}
    if kind == "expv":
        s["opt"] = dict(m=case["m"], tol=case["tol"], iop=case["q"] > 0, q_iop=max(1, case["q"]), coefs=m.coefs(0.0))
    else:
        s["B"] = BDFIntegrator(A, rtol=case["rtol"], atol=case["atol"])
    return s


def run(s):
    kind = s["kind"]
    if kind == "action":
        s["A"].action(s["t"], s["x"], s["y"])
        return s["y"]
    if kind == "transpose":
        s["A"].apply_transpose(s["x"], s["y"], coefs=s["c"])
        return s["y"]
    if kind == "gradient":
        ll, g = s["L"].gradient(s["c"])
        return [ll, g]
    p = s["p"]
    if kind == "batch":
        p.copy_(s["p0"])
        s["B"].solve(s["t"], p)
    elif kind == "expv":
        p.copy_(s["p0"])
        KryExpvFSP(s["t"], s["A"], p, **s["opt"]).solve()
    else:
        s["B"].init(0.0, s["p0"])
        s["B"].advance(s["t"], p)
    return p


# ---- work ------------------------------------------------------------------------------------------

def _rate_bound(m):
    """Largest total outflow of a state, bounded reaction by reaction."""
    tot, c = 0.0, np.maximum(m.coefs(0.0), m.rates)
    for r in range(m.nr):
        f, off = c[r], 0
        for b in m.bounds:
            f *= float(np.max(m.tables[r, off:off + b + 1]))
            off += b + 1
        tot += f
    return tot


def _applications(m, t, tol):
    """Generator applications that a polynomial method needs at least for exp(tA) p."""
    return max(1, math.ceil(math.sqrt(_rate_bound(m) * t * math.log(1.0 / tol))))


def work(case):
    """Inputs read once and outputs written once; one multiply-add per state and reaction for the gain
    and one for the outflow of each generator application the path cannot do without."""
    kind = case["kind"]
    if kind == "batch":
        ms = _batch_models(case, 1)
        n = sum(m.n_states for m in ms)
        return {"bytes": 16.0 * n, "flops": sum(4.0 * m.nr * m.n_states * _applications(m, case["t"], case["tol"]) for m in ms)}
    m = _model(case, 1)
    n, nr = m.n_states, m.nr
    if kind == "action":
        return {"bytes": (24.0 + (0.0 if case["format"] == "kron" else 8.0 * nr)) * n, "flops": 4.0 * nr * n}
    if kind == "transpose":
        return {"bytes": 16.0 * n, "flops": 4.0 * nr * n}
    tol = case["rtol"] if kind == "bdf" else case["tol"]
    a = _applications(m, case["t"], tol)
    if kind == "gradient":
        return {"bytes": 8.0 * n + 8.0 * case["times"] * n / 8 + 8.0 * (nr + 1), "flops": 2 * 4.0 * nr * n * a}
    return {"bytes": 16.0 * n, "flops": 4.0 * nr * n * a}


# ---- the same results in plain torch ----------------------------------------------------------------

class _Generator:
    """sum_r c_r A_r on a box as torch slices: species 0 is the fastest axis, so axis -1.  Vectors may
    carry leading axes."""

    def __init__(self, bounds, nu, tables):
        self.shape = tuple(b + 1 for b in reversed(bounds))
        ns, nr = len(bounds), nu.shape[0]
        self.a, self.dst, self.src = [], [], []
        for r in range(nr):
            f, off = torch.ones((), dtype=torch.float64, device="cuda"), 0
            d, s = [Ellipsis], [Ellipsis]
            for k, b in enumerate(bounds):
                t = torch.as_tensor(tables[r, off:off + b + 1], device="cuda")
                f = f * t.reshape([-1 if ns - 1 - j == k else 1 for j in range(ns)])
                off += b + 1
            for k in reversed(range(ns)):
                v, size = int(nu[r, k]), bounds[k] + 1
                d.append(slice(max(v, 0), size + min(v, 0)))
                s.append(slice(max(-v, 0), size + min(-v, 0)))
            self.a.append(f.expand(self.shape).contiguous())
            self.dst.append(tuple(d))
            self.src.append(tuple(s))

    def one(self, r, x):
        """A_r x at unit rate."""
        g = self.a[r] * x
        y = -g
        y[self.dst[r]] += g[self.src[r]]
        return y

    def one_t(self, r, x):
        y = -x
        y[self.src[r]] += x[self.dst[r]]
        return y.mul_(self.a[r])

    def apply(self, c, x, transpose=False):
        y = torch.zeros_like(x)
        for r in range(len(self.a)):
            y.add_((self.one_t if transpose else self.one)(r, x), alpha=float(c[r]))
        return y

    def outflow(self, c):
        return sum(float(c[r]) * self.a[r] for r in range(len(self.a)))

    def exp(self, c, t, x, force=None):
        """exp(t A) x by uniformisation: every term is non-negative for non-negative x.  With force(x) =
        the right-hand side fed from x[0] into the leading axis, the exponential of that larger system."""
        out = self.outflow(c)
        lam = float(out.max()) * 1.0001 + 1e-300
        stay = 1.0 - out / lam
        gain = [self.a[r] * (float(c[r]) / lam) for r in range(len(self.a))]
        del out
        parts = max(1, math.ceil(lam * t / 200.0))
        mu = lam * t / parts
        terms = int(mu + 9.0 * math.sqrt(mu) + 40.0)
        for _ in range(parts):
            w = math.exp(-mu)
            acc, cur = x * w, x
            for k in range(1, terms):
                nxt = cur * stay
                for r in range(len(gain)):
                    nxt[self.dst[r]] += gain[r][self.src[r]] * cur[self.src[r]]
                if force is not None:
                    force(cur, nxt, lam)
                cur = nxt
                w *= mu / k
                acc.add_(cur, alpha=w)
            x = acc
        return x


def _exact_gradient(case, seed, m):
    """log L and d log L / d log c by forward sensitivities z_r' = A z_r + A_r p beside p' = A p."""
    G, c = _Generator(m.bounds, m.nu, m.tables), m.coefs(0.0)
    counts = torch.as_tensor(_counts(case, seed, m.bounds), device="cuda")
    x = torch.zeros((m.nr + 1,) + G.shape, dtype=torch.float64, device="cuda")
    x[0].view(-1)[0] = 1.0
    ll, grad, prev = 0.0, torch.zeros(m.nr, dtype=torch.float64, device="cuda"), 0.0

    def force(cur, nxt, lam):
        for r in range(m.nr):
            g = G.a[r] * cur[0]
            nxt[r + 1].sub_(g, alpha=1.0 / lam)
            nxt[r + 1][G.dst[r]] += g[G.src[r]] / lam

    for i, t in enumerate(_times(case)):
        x = G.exp(c, t - prev, x, force)
        prev = t
        q = x.reshape(m.nr + 1, -1, 8).sum(-1)
        ll += float((counts[i] * torch.log(q[0].clamp_min(1e-44))).sum())
        ratio = torch.where((counts[i] > 0) & (q[0] > 1e-44), counts[i] / q[0], torch.zeros_like(q[0]))
        grad += (q[1:] * ratio).sum(-1)
    return [ll, grad.cpu().numpy() * c]


def _exact_bdf(case, seed, m):
    """Classical fourth-order Runge-Kutta with steps far below the accuracy of the integrator's."""
    G = _Generator(m.bounds, m.nu, m.tables)
    x = _start(case, seed, m.bounds).reshape(G.shape)
    steps = math.ceil(case["t"] * max(400.0, 3.0 * _rate_bound(m)))
    h = case["t"] / steps
    for k in range(steps):
        t = k * h
        c0, c1, c2 = m.coefs(t), m.coefs(t + 0.5 * h), m.coefs(t + h)
        k1 = G.apply(c0, x)
        k2 = G.apply(c1, x + 0.5 * h * k1)
        k3 = G.apply(c1, x + 0.5 * h * k2)
        k4 = G.apply(c2, x + h * k3)
        x = x + (h / 6.0) * (k1 + 2.0 * (k2 + k3) + k4)
    return x.reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        out = []
        for i, m in enumerate(_batch_models(case, seed)):
            G = _Generator(m.bounds, m.nu, m.tables)
            p = G.exp(m.coefs(0.0), case["t"], _start(case, seed + i, m.bounds).reshape(G.shape)).reshape(-1)
            out.append(torch.nn.functional.pad(p, (0, m.n_states % 2)))
        return torch.cat(out)
    m = _model(case, seed)
    if kind == "gradient":
        return _exact_gradient(case, seed, m)
    if kind == "bdf":
        return _exact_bdf(case, seed, m)
    G = _Generator(m.bounds, m.nu, m.tables)
    if kind == "expv":
        return G.exp(m.coefs(0.0), case["t"], _start(case, seed, m.bounds).reshape(G.shape)).reshape(-1)
    x, y = _vectors(case, seed, m.n_states)
    x = x.reshape(G.shape)
    if kind == "transpose":
        return G.apply(m.coefs(0.0), x, transpose=True).reshape(-1)
    return y + G.apply(m.coefs(1.0), x).reshape(-1)
