"""The work that users of ennemi_gb300 have it do, as measurable cases.

A case names a ``family`` (one way of calling the framework), its sizes and
its options:

  mi        estimate_mi of one pair: the quick-start call, the single
            10,000-sample estimate, large samples, large k
  lags      estimate_mi over several variables and lags, with a condition, a
            mask or dropped NaNs: time-series exploration
  pairwise  pairwise_mi / pairwise_corr of a table of variables, plain or
            given a condition
  semi      Ross MI of continuous columns against class labels, one batch
  entropy   estimate_entropy of a multidimensional variable
  discrete  estimate_mi of two discrete variables
  points    the two neighbour queries alone (knn_eps, ball_count)
  device    one batch of estimates on device-resident columns (run_tasks)

Inputs are host NumPy arrays, as in the reference's own use, except for the
``device`` family.  All values come from the case's seed.
"""

import math

import numpy as np
import torch

import ennemi_gb300 as ennemi
from ennemi_gb300 import _entropy_estimators as estimators
from ennemi_gb300 import _native

EPS_SHIFT = 1e-12                 # counts use the radius eps - 1e-12
NOISE_SEED = 2_718281828          # the preprocessing noise of estimate_mi


def listed():
    return [
        # the quick-start call: one pair of a few hundred observations
        {"name": "mi-400", "family": "mi", "n": 400, "k": 3, "rho": 0.6},
        # lag search on a short series given a condition (three coupled
        # series of 1,000 samples, lags on both sides of zero)
        {"name": "cmi-lags-1k", "family": "lags", "n": 1000, "nx": 2, "lag0": -10, "nlag": 21,
         "dz": 1, "mask": False, "nan": False, "k": 3},
        # the single estimate of the plain KSG configuration
        {"name": "mi-10k", "family": "mi", "n": 10_000, "k": 3, "rho": 0.6},
        # the large-k estimate of the large-sample benchmark (k = 50, 20,000
        # samples): less variance, more neighbours
        {"name": "mi-20k-k50", "family": "mi", "n": 20_000, "k": 50, "rho": 0.6},
        # measured series with gaps: every task keeps its own rows
        {"name": "lags-nan-20k", "family": "lags", "n": 20_011, "nx": 4, "lag0": 0, "nlag": 13,
         "dz": 0, "mask": False, "nan": True, "k": 3},
        # partial correlations of a table given two shared conditions
        {"name": "pairwise-cond-16x20k", "family": "pairwise", "n": 20_000, "nvar": 16, "dz": 2,
         "k": 3, "corr": True},
        # the neighbour queries alone, three columns, an odd count
        {"name": "points-100k-3d", "family": "points", "n": 100_003, "d": 3, "k": 5},
        # entropy of one three-dimensional variable
        {"name": "entropy-3d-200k", "family": "entropy", "n": 200_000, "d": 3, "k": 3},
        # class labels against 1 to 4 continuous columns, uneven classes
        {"name": "semi-500k", "family": "semi", "n": 500_000, "d": 4, "classes": 25, "k": 3},
        # the large-sample batch: four pairs and one conditional estimate of
        # a million samples each, already on the device
        {"name": "device-1m", "family": "device", "n": 1_000_000, "npair": 4, "ncond": 1, "k": 3},
        # 16 coupled series of 200,000 samples, lags 0..48, a tenth masked
        {"name": "lags-200k", "family": "lags", "n": 200_000, "nx": 16, "lag0": 0, "nlag": 49,
         "dz": 0, "mask": True, "nan": False, "k": 3},
        # every pair of 64 mixed variables (Gaussian, sine, heavy tails)
        {"name": "pairwise-64x50k", "family": "pairwise", "n": 50_000, "nvar": 64, "dz": 0, "k": 3,
         "corr": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["mi", "mi", "lags", "lags", "pairwise", "semi", "entropy", "discrete", "points",
                         "device"])
    k = rng.choice([1, 2, 3, 3, 3, 4, 5, 7, 8, 12])
    if family == "mi":
        if rng.random() < 0.25:   # large k: moderate samples
            return {"family": family, "n": _log(rng, 500, 30_000), "k": rng.randint(20, 100),
                    "rho": round(rng.uniform(-0.95, 0.95), 3)}
        return {"family": family, "n": _log(rng, 100, 1_000_000), "k": k,
                "rho": round(rng.uniform(-0.95, 0.95), 3)}
    if family == "lags":
        n = _log(rng, 200, 100_000)
        nan = rng.random() < 0.25
        return {"family": family, "n": n, "nx": rng.randint(1, 6), "lag0": rng.randint(-12, 4),
                "nlag": rng.randint(1, 16), "dz": rng.choice([0, 0, 1, 1, 2]),
                "mask": rng.random() < 0.5, "nan": nan, "k": k}
    if family == "pairwise":
        return {"family": family, "n": _log(rng, 300, 30_000), "nvar": rng.randint(3, 20),
                "dz": rng.choice([0, 0, 1, 2]), "k": rng.choice([2, 3, 3, 4, 5]),
                "corr": rng.random() < 0.5}
    if family == "semi":
        return {"family": family, "n": _log(rng, 500, 300_000), "d": rng.randint(1, 4),
                "classes": rng.randint(2, 40), "k": rng.choice([2, 3, 3, 5])}
    if family == "entropy":
        return {"family": family, "n": _log(rng, 200, 500_000), "d": rng.randint(1, 4), "k": k}
    if family == "discrete":
        return {"family": family, "n": _log(rng, 200, 500_000), "levels": _log(rng, 2, 40)}
    if family == "points":
        return {"family": family, "n": _log(rng, 300, 300_000), "d": rng.randint(1, 5), "k": k}
    return {"family": family, "n": _log(rng, 5_000, 1_000_000), "npair": rng.randint(1, 4),
            "ncond": rng.randint(0, 2), "k": rng.choice([2, 3, 3, 4, 5])}


# --------------------------------------------------------------- inputs --

def _coupled_series(rng, n, m):
    """m coupled AR(1) series: x_i(t) = .8 x_i(t-1) + .3 x_{i-1}(t-5) + e."""
    out = np.empty((n, m))
    for i in range(m):
        s = rng.standard_normal(n)
        if i:
            s[5:] += 0.3 * out[:-5, i - 1]
        a, step = 0.8, 1
        while step < min(n, 256):   # s <- sum_j .8^j s(t - j), doubling the span
            t = s.copy()
            t[step:] += a * s[:-step]
            s, a, step = t, a * a, 2 * step
        out[:, i] = s
    return out


def _runs(rng, n, share):
    """A boolean array with about `share` true, in runs of 1 to 50."""
    hit = np.zeros(n, dtype=bool)
    starts = rng.integers(0, n, max(1, int(share * n / 25)))
    for s, r in zip(starts, rng.integers(1, 51, len(starts))):
        hit[s:s + r] = True
    return hit


def _table(rng, n, m):
    """m mixed columns: correlated Gaussian, noisy sine, Student t(3), log-normal."""
    base = rng.standard_normal((n, m))
    common = rng.standard_normal(n)
    out = np.empty((n, m))
    for c in range(m):
        kind = c % 4
        if kind == 0:
            out[:, c] = 0.7 * base[:, c] + 0.5 * common
        elif kind == 1:
            out[:, c] = np.sin(2 * base[:, c]) + 0.3 * rng.standard_normal(n)
        elif kind == 2:
            chi = sum(rng.standard_normal(n) ** 2 for _ in range(3))
            out[:, c] = base[:, c] / np.sqrt(chi / 3)
        else:
            out[:, c] = np.exp(base[:, c])
    return out


def _mixture(rng, n, d):
    """A mixture of three d-dimensional Gaussians."""
    comp = rng.integers(0, 3, n)
    mean = rng.normal(scale=2.0, size=(3, d))
    scale = rng.uniform(0.5, 1.5, size=(3, d))
    x = rng.standard_normal((n, d)) * scale[comp] + mean[comp]
    x[:, 1:] += 0.4 * x[:, :1]
    return x


def prepare(case, seed):
    rng = np.random.default_rng([seed, case["n"]])
    family, n = case["family"], case["n"]
    s = {"case": case}
    if family == "mi":
        x = rng.standard_normal(n)
        rho = case["rho"]
        s["x"], s["y"] = x, rho * x + math.sqrt(1 - rho * rho) * rng.standard_normal(n)
    elif family == "lags":
        nx, dz = case["nx"], case["dz"]
        series = _coupled_series(rng, n, nx + dz)
        s["x"] = np.ascontiguousarray(series[:, :nx])
        s["y"] = series[:, 0] + 0.5 * rng.standard_normal(n) if nx + dz < 8 else series[:, 0].copy()
        s["lag"] = np.arange(case["lag0"], case["lag0"] + case["nlag"])
        s["z"] = np.ascontiguousarray(series[:, nx:]) if dz else None
        s["mask"] = ~_runs(rng, n, 0.1) if case["mask"] else None
        if case["nan"]:
            for c in range(nx):
                s["x"][_runs(rng, n, 0.02), c] = np.nan
    elif family == "pairwise":
        s["x"] = _table(rng, n, case["nvar"])
        s["z"] = rng.standard_normal((n, case["dz"])) if case["dz"] else None
        if case["dz"]:
            s["x"] += 0.3 * s["z"][:, :1]
    elif family == "semi":
        s["tasks"], s["data"] = [], []
        for d in range(1, case["d"] + 1):
            p = rng.dirichlet(np.full(case["classes"], 0.5)) * 0.9 + 0.1 / case["classes"]
            y = rng.choice(case["classes"], p=p, size=n)
            x = _mixture(rng, n, d) + (0.5 * y / case["classes"])[:, None]
            x = x if d > 1 else x[:, 0].copy()
            s["data"].append((x, y))
            s["tasks"].append(estimators.semidiscrete_task(x, y, case["k"]))
    elif family == "entropy":
        s["x"] = _mixture(rng, n, case["d"])
    elif family == "discrete":
        s["x"] = rng.integers(0, case["levels"], n)
        s["y"] = (s["x"] + rng.integers(0, 3, n)) % case["levels"]
    elif family == "points":
        s["x"] = _mixture(rng, n, case["d"])
        s["r"] = rng.uniform(0.2, 1.0, n) * n ** (-1.0 / (case["d"] + 1))
    elif family == "device":
        s["columns"] = []
        for t in range(case["npair"] + case["ncond"]):
            rho = (0.0, 0.3, 0.6, 0.9)[t % 4] if t < case["npair"] else 0.5
            x = rng.standard_normal(n)
            y = rho * x + math.sqrt(1 - rho * rho) * rng.standard_normal(n)
            cols = [x, y]
            if t >= case["npair"]:
                cols.append(0.3 * (x + y) + rng.standard_normal(n))
            s["columns"].append([torch.from_numpy(c).cuda() for c in cols])
        s["tasks"] = [_native.Task(_native.MI if len(c) == 2 else _native.CMI, case["k"], [c[0]], [c[1]],
                                   [c[2]] if len(c) == 3 else (), n=n) for c in s["columns"]]
    return s


# ----------------------------------------------------------------- run --

def run(state):
    case = state["case"]
    family, k = case["family"], case.get("k", 3)
    if family == "mi":
        return ennemi.estimate_mi(state["y"], state["x"], k=k)
    if family == "lags":
        return ennemi.estimate_mi(state["y"], state["x"], state["lag"], k=k, cond=state["z"],
                                  mask=state["mask"], drop_nan=case["nan"])
    if family == "pairwise":
        call = ennemi.pairwise_corr if case["corr"] else ennemi.pairwise_mi
        return call(state["x"], k=k, cond=state["z"])
    if family == "semi":
        return _native.run_tasks(state["tasks"])
    if family == "entropy":
        return ennemi.estimate_entropy(state["x"], k=k, multidim=True)
    if family == "discrete":
        return ennemi.estimate_mi(state["y"], state["x"], discrete_x=True, discrete_y=True)
    if family == "points":
        return {"eps": _native.knn_eps(state["x"], k), "count": _native.ball_count(state["x"], state["r"])}
    return _native.run_tasks(state["tasks"], flags=_native.INPUT_DEVICE)


# ---------------------------------------------------------------- work --

def _tasks(case):
    """(number of estimates, columns searched by each)."""
    f = case["family"]
    if f == "lags":
        return case["nx"] * case["nlag"], 2 + case["dz"]
    if f == "pairwise":
        return case["nvar"] * (case["nvar"] - 1) // 2, 2 + case["dz"]
    if f == "semi":
        return case["d"], (case["d"] + 1) / 2
    if f == "device":
        return case["npair"] + case["ncond"], 2
    return 1, case.get("d", 2)


def work(case):
    """Bytes: every input and output once.  Operations: one ordered search
    (log2 n comparisons) per sample, column and estimate."""
    n, f = case["n"], case["family"]
    tasks, cols = _tasks(case)
    inputs = {"lags": case.get("nx", 0) + 1 + case.get("dz", 0), "pairwise": case.get("nvar", 0) + case.get("dz", 0),
              "semi": tasks * (cols + 0.5), "device": 2 * tasks + case.get("ncond", 0),
              "points": cols + 1, "entropy": cols}.get(f, 2)
    outputs = 2 * n if f == "points" else case["nvar"] ** 2 if f == "pairwise" else tasks
    return {"bytes": 8.0 * (n * inputs + outputs), "flops": float(tasks * cols * n * max(1.0, math.log2(n)))}


# --------------------------------------------------------------- exact --

_PAIRS = 6e10   # point pairs that brute force gets through in a few seconds


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _psi(v):
    """Digamma of integers >= 1 by the estimator's asymptotic expansion."""
    v = v.double()
    v2 = v * v
    e = torch.log(v) - v ** -6 * (v2 * (v2 * (v / 2 + 1 / 12) - 1 / 120) + 1 / 252)
    return torch.where(v == 1, torch.full_like(v, -0.5772156649015331), e)


def _blocks(n):
    step = max(1, int(2e8) // n)
    return [(a, min(a + step, n)) for a in range(0, n, step)]


def _dist(cols, a, b):
    d = None
    for c in cols:
        t = (c[a:b, None] - c[None, :]).abs_()
        d = t if d is None else torch.maximum(d, t)
    return d


def _knn(cols, k):
    n = len(cols[0])
    out = [torch.topk(_dist(cols, a, b), k + 1, dim=1, largest=False).values[:, -1] for a, b in _blocks(n)]
    return torch.cat(out)


def _count(cols, r):
    n = len(cols[0])
    return torch.cat([(_dist(cols, a, b) <= r[a:b, None]).sum(1) for a, b in _blocks(n)])


def _mi(x, y, z, k):
    """KSG MI, or the conditional estimate given the columns z."""
    n = len(x)
    r = _knn([x, y] + z, k) - EPS_SHIFT
    one = torch.ones(1, dtype=torch.float64, device=x.device)
    if not z:
        m = (_psi(_count([x], r)) + _psi(_count([y], r))).mean()
        return float(_psi(one * n) + _psi(one * k) - m)
    m = (_psi(_count([x] + z, r)) + _psi(_count([y] + z, r)) - _psi(_count(z, r))).mean()
    return float(_psi(one * k) - m)


def _scaled(x, y, z):
    """Unit variance plus the fixed-seed 1e-10 noise, drawn in the order x, y, z."""
    rng = np.random.default_rng(NOISE_SEED)
    cols = []
    for v in (x, y) if z is None else (x, y, z):
        v = (v - v.mean(axis=0)) / v.std(axis=0)
        cols.append(v + rng.normal(0.0, 1e-10, v.shape))
    dev = _device()
    x, y = (torch.from_numpy(c).to(dev) for c in cols[:2])
    z = [torch.from_numpy(np.ascontiguousarray(c)).to(dev) for c in cols[2].T] if z is not None else []
    return x, y, z


def exact(case, seed):
    family, n, k = case["family"], case["n"], case.get("k", 3)
    if family != "discrete" and _tasks(case)[0] * float(n) ** 2 > _PAIRS:
        return None
    s = prepare(case, seed)
    dev = _device()
    if family == "mi":
        return np.array([[_mi(*_scaled(s["x"], s["y"], None), k)]])
    if family == "lags":
        lo, hi = min(int(s["lag"].min()), 0), max(int(s["lag"].max()), 0)
        out = np.empty((len(s["lag"]), case["nx"]))
        for i, lag in enumerate(s["lag"]):
            for j in range(case["nx"]):
                x = s["x"][hi - lag: n - lag + lo, j]
                y = s["y"][hi: n + lo]
                z = None if s["z"] is None else s["z"][hi: n + lo]
                keep = np.ones(len(y), dtype=bool) if s["mask"] is None else s["mask"][hi: n + lo].copy()
                keep &= ~(np.isnan(x) | np.isnan(y))
                out[i, j] = _mi(*_scaled(x[keep], y[keep], None if z is None else z[keep]), k)
        return out
    if family == "pairwise":
        m = case["nvar"]
        out = np.full((m, m), np.nan)
        for i in range(m):
            for j in range(i + 1, m):
                v = _mi(*_scaled(s["x"][:, i], s["x"][:, j], s["z"]), k)
                if case["corr"] and v > 0:
                    v = math.sqrt(1 - math.exp(-2 * v))
                out[i, j] = out[j, i] = v
        return out
    one = torch.ones(1, dtype=torch.float64, device=dev)
    if family == "semi":
        out = []
        for x, y in s["data"]:
            cols = [torch.from_numpy(np.ascontiguousarray(c)).to(dev) for c in x.reshape(n, -1).T]
            lab = torch.from_numpy(y).to(dev)
            r = torch.empty(n, dtype=torch.float64, device=dev)
            w = 0.0
            for c in np.unique(y):
                at = torch.nonzero(lab == int(c)).ravel()
                m = len(at)
                r[at] = _knn([v[at] for v in cols], k) - EPS_SHIFT if m > k else math.inf
                w += float(_psi(one * m)) * m / n
            out.append(float(_psi(one * n) + _psi(one * k) - _psi(_count(cols, r)).mean()) - w)
        return np.array(out)
    if family == "discrete":
        joint = np.zeros((case["levels"], case["levels"]))
        np.add.at(joint, (s["x"], s["y"]), 1.0)
        px, py = joint.sum(1), joint.sum(0)
        a, b = np.nonzero(joint)
        j = joint[a, b]
        return np.array([[float(np.sum(j * np.log(n * j / (px[a] * py[b]))) / n)]])
    if family == "device":
        return np.array([_mi(c[0].to(dev), c[1].to(dev), [v.to(dev) for v in c[2:]], k) for c in s["columns"]])
    cols = [torch.from_numpy(np.ascontiguousarray(c)).to(dev) for c in s["x"].T]
    eps = _knn(cols, k)
    if family == "entropy":
        d = len(cols)
        return np.asarray(float(_psi(one * n) - _psi(one * k) + d * (torch.log(eps).mean() + math.log(2.0))))
    r = torch.from_numpy(s["r"]).to(dev)
    return {"eps": eps.cpu().numpy(), "count": _count(cols, r).cpu().numpy()}
