"""Timing cases: what a user of this framework has it do, through its public
entry points.

A user fits a Gaussian process: once per data set the conditioning sets are
selected on the device (`knn`), then an optimizer asks for one block-Vecchia
log-likelihood after another (`LlhData`, `eval_host` when the observations
come from the host each time, `Server` when several fits share the device).

Kinds of case:
  eval    one log-likelihood of a resident layout at one parameter vector
  host    the same from host observations (simulation studies)
  knn     conditioning-set selection, host arrays in and out
  serve   one request of each of several concurrent fitting jobs

The layouts are made here (blocks of neighbouring points, random block order,
the first blocks merged until they hold cs points, as the driver's layout
steps do) so that each seed's inputs are made quickly.
"""
import math
import random

import numpy as np
import torch

import blockvecchia_b200 as bv

# Half-smooth fields (nu = 1/2, 3/2, 5/2) have closed forms; an optimizer's
# probes have any nu.  Smooth fields with a general nu are left out: their
# covariances are singular to working precision, so no value is comparable.


def listed():
    return [
        # The smallest fit: the layout the tests use; latency counts.
        dict(name="eval-2k", kind="eval", n=2000, bs=13, cs=60, nu=1.5, range=0.08, sigma2=1.0),
        # Classic Vecchia: one point per block, small conditioning sets.
        dict(name="eval-classic-30k", kind="eval", n=30011, bs=1, cs=30, nu=0.5, range=0.1, sigma2=1.5),
        # The small configuration: large conditioning sets, exponential kernel.
        dict(name="eval-20k-cs300", kind="eval", n=20000, bs=13, cs=300, nu=0.5, range=0.1, sigma2=1.5),
        # The batching configuration: uneven blocks of 3-30 points.
        dict(name="eval-200k-cs120", kind="eval", n=200000, bs=10, cs=120, nu=1.5, range=0.08, sigma2=1.0),
        # The headline configuration (some pivots fail in any FP64 evaluation
        # at this smoothness and density: the value skips them).
        dict(name="eval-1m-cs200", kind="eval", n=1000000, bs=10, cs=200, nu=2.5, range=0.05, sigma2=1.0),
        # An optimizer's probe of the batching configuration's size, nu free.
        dict(name="probe-100k-cs120", kind="eval", n=100003, bs=10, cs=120, nu=0.8, range=0.1, sigma2=0.9),
        # The general-nu configuration: clustered locations, nugget, cs = 300.
        dict(name="probe-mixture-200k-cs300", kind="eval", n=200000, bs=10, cs=300, nu=0.8, range=0.1,
             sigma2=1.0, nugget=0.01, locations="mixture"),
        # Space-time fit: the separable-in-form kernel over 20 time slots.
        dict(name="spacetime-20k-cs100", kind="eval", n=20000, bs=8, cs=100, nu=0.5, range=0.1, sigma2=1.0,
             slots=20),
        # Simulation study: new host observations for every evaluation.
        dict(name="host-50k-cs60", kind="host", n=50021, bs=10, cs=60, nu=1.5, range=0.05, sigma2=1.0),
        # Conditioning sets of the small and of the headline configuration.
        dict(name="knn-20k-cs300", kind="knn", n=20000, bs=13, cs=300),
        dict(name="knn-1m-cs200", kind="knn", n=1000000, bs=10, cs=200),
        # Ten concurrent fitting jobs of mixed sizes, one request each.
        dict(name="serve-10", kind="serve", jobs=10, n_min=5000, n_max=60000),
    ]


def _loguniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """A case of the ranges the listed ones span."""
    kind = rng.choice(["eval", "eval", "eval", "eval", "host", "knn", "serve"])
    if kind == "serve":
        n_min = int(_loguniform(rng, 3000, 8000))
        return dict(kind=kind, jobs=rng.randint(4, 10), n_min=n_min,
                    n_max=n_min * rng.randint(3, 8) + rng.randint(0, 999))
    bs = rng.randint(4, 16)
    cs = rng.choice([20, 30, 47, 60, 100, 120, 150, 200, 231, 300])
    if kind == "knn":
        c = dict(kind=kind, n=int(_loguniform(rng, 3000, 1000000)), bs=bs, cs=cs)
        if rng.random() < 0.3:
            c["locations"] = "mixture"
        return c
    # Work grows as (n / bs) (cs + bs)^3: stay below the headline's.
    cap = 1.0e12 * bs / float(cs + 2 * bs) ** 3
    n = int(_loguniform(rng, 2000, min(1000000.0, cap)))
    if kind == "host":
        return dict(kind=kind, n=min(n, 300000), bs=bs, cs=min(cs, 120), nu=rng.choice([0.5, 1.5]),
                    range=round(rng.uniform(0.02, 0.08), 4), sigma2=round(rng.uniform(0.5, 2.0), 3))
    c = dict(kind=kind, bs=bs, cs=cs, sigma2=round(rng.uniform(0.5, 2.0), 3))
    form = rng.random()
    if form < 0.55:  # closed forms
        c.update(n=n, nu=rng.choice([0.5, 0.5, 1.5]), range=round(rng.uniform(0.02, 0.1), 4))
    elif form < 0.85:  # a probe
        c.update(n=min(n, 300000), nu=round(rng.uniform(0.4, 1.2), 3), range=round(rng.uniform(0.02, 0.1), 4))
        if rng.random() < 0.5:
            c["nugget"] = round(_loguniform(rng, 0.001, 0.1), 5)
            if rng.random() < 0.5:
                c["locations"] = "mixture"
    else:
        c.update(n=min(n, 60000), nu=0.5, range=round(rng.uniform(0.05, 0.15), 4), slots=rng.randint(5, 30))
    return c


# ------------------------------------------------------------------ inputs

def _locations(case, g):
    n = case["n"]
    if case.get("slots"):
        t = case["slots"]
        m = -(-n // t)
        x, y = np.tile(g.random(m), t)[:n], np.tile(g.random(m), t)[:n]
        # Stations that report once per slot at times of their own: times in
        # common leave near-ties at the cs-th distance, whose order only the
        # framework's own key arithmetic decides.
        return x, y, (np.repeat(np.arange(t), m)[:n] + g.random(n)) / t
    if case.get("locations") == "mixture":
        k = 50
        centers, stds = g.random((k, 2)), g.uniform(0.01, 0.05, k)
        comp = g.integers(0, k, n)
        p = centers[comp] + g.standard_normal((n, 2)) * stds[comp, None]
        return p[:, 0].copy(), p[:, 1].copy(), None
    return g.random(n), g.random(n), None


def _observations(x, y, z, case, g):
    """A draw of a Matern process by random Fourier features (in time: a
    rough process of the same form)."""
    f = 128
    nu = min(case.get("nu", 0.5), 2.5)
    scale = case.get("range", 0.1) * np.sqrt(g.chisquare(2 * nu, f))
    om = g.standard_normal((f, 2)) / scale[:, None]
    ph = g.random(f) * 2 * np.pi
    oz = g.standard_cauchy(f) * 2.0
    amp = math.sqrt(2 * case.get("sigma2", 1.0) / f)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    to = lambda a: torch.as_tensor(a, device=dev)  # noqa: E731
    X, Y, O, P = to(x), to(y), to(om), to(ph)
    Z, OZ = (to(z), to(oz)) if z is not None else (None, None)
    out = torch.empty(len(x), dtype=torch.float64, device=dev)
    for s in range(0, len(x), 131072):
        e = s + 131072
        a = X[s:e, None] * O[:, 0] + Y[s:e, None] * O[:, 1] + P
        if Z is not None:
            a = a + Z[s:e, None] * OZ
        out[s:e] = torch.cos(a).sum(1) * amp
    obs = out.cpu().numpy()
    if case.get("nugget"):
        obs = obs + math.sqrt(case["nugget"]) * g.standard_normal(len(x))
    return obs


def _layout(case, seed):
    """Locations, observations and blocks of neighbouring points."""
    n, bs, cs = case["n"], case["bs"], case["cs"]
    g = np.random.default_rng([int(seed), 77])
    shape = np.random.default_rng([n, bs, cs])  # block sizes and order: the case's, not the seed's
    x, y, z = _locations(case, g)
    obs = _observations(x, y, z, case, g)
    # Strips in x, then (for a third coordinate) slabs of a few time slots,
    # cut along y into blocks of uneven sizes.
    dims = 2 if z is None else 3
    strips = max(1, int(round((n / bs) ** (1.0 / dims))))
    rank = np.empty(n, dtype=np.int64)
    rank[np.argsort(x, kind="stable")] = np.arange(n)
    key = rank * strips // n
    if z is not None:
        zr = np.empty(n, dtype=np.int64)
        zr[np.argsort(z, kind="stable")] = np.arange(n)
        slabs = max(1, min(strips, case["slots"]))
        key = key * slabs + zr * slabs // n
    order = np.lexsort((y, key))
    if bs == 1:
        label_sizes = np.ones(n, dtype=np.int64)
    else:
        sizes = shape.integers(max(1, bs // 3), 2 * bs - bs // 3 + 1, 2 * n // bs + 16)
        cut = int(np.searchsorted(np.cumsum(sizes), n))
        label_sizes = sizes[:cut + 1].copy()
        label_sizes[-1] -= int(label_sizes.sum()) - n
    k = len(label_sizes)
    starts = np.concatenate([[0], np.cumsum(label_sizes)])
    perm = shape.permutation(k)  # random block order
    merged = int(np.searchsorted(np.cumsum(label_sizes[perm]), cs)) + 1  # first block: >= cs points
    bsz = label_sizes[perm]
    src = np.repeat(starts[:-1][perm], bsz) + (np.arange(n) - np.repeat(np.cumsum(bsz) - bsz, bsz))
    idx = order[src]
    batch = np.concatenate([[bsz[:merged].sum()], bsz[merged:]]).astype(np.int32)
    acc = np.concatenate([[0], np.cumsum(batch)]).astype(np.int32)
    mean = lambda v: np.add.reduceat(v[idx], acc[:-1]) / batch  # noqa: E731
    return bv.Layout(batch, acc, x[idx], y[idx], obs[idx], cs, mean(x), mean(y),
                     z=None if z is None else z[idx], cz=None if z is None else mean(z))


def _theta(case):
    if case.get("slots"):
        return (case["sigma2"], case["range"], case["nu"], 0.5, 0.9, 0.7, 0.0)
    th = (case["sigma2"], case["range"], case["nu"])
    return th + ((case["nugget"],) if case.get("nugget") else ())


def _jobs(case, seed):
    r = random.Random(1000 + case["jobs"])
    out = []
    for j in range(case["jobs"]):
        # The first and last job have the range's ends as their sizes.
        n = (case["n_min"] if j == 0 else case["n_max"] if j == case["jobs"] - 1
             else int(_loguniform(r, case["n_min"], case["n_max"])))
        c = dict(n=n, bs=10, cs=(60, 120, 300)[j % 3], nu=(0.5, 0.8, 1.5, 1.1)[j % 4],
                 range=round(r.uniform(0.02, 0.1), 4), sigma2=round(r.uniform(0.5, 2.0), 3))
        out.append((c, int(seed) * 64 + j))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "serve":
        srv = bv.Server(device=0, hbm_budget=8 << 30)
        jobs = []
        for c, s in _jobs(case, seed):
            L = _layout(c, s)
            L.knn_idx = bv.knn(L)
            jobs.append((srv.open_job(L), _theta(c)))
        return dict(kind=kind, server=srv, jobs=jobs)
    L = _layout(case, seed)
    if kind == "knn":
        return dict(kind=kind, layout=L)
    L.knn_idx = bv.knn(L)
    st = dict(kind=kind, theta=_theta(case),
              data=bv.LlhData(L, kernel=4 if case.get("slots") else 1, nugget=bool(case.get("nugget")),
                              on_failure="continue"))
    if kind == "host":
        st["obs"] = torch.from_numpy(L.obs).pin_memory().numpy()
    return st


def run(state):
    kind = state["kind"]
    if kind == "eval":
        return np.float64(state["data"](state["theta"]))
    if kind == "host":
        return np.float64(state["data"].eval_host(state["obs"], state["theta"]))
    if kind == "knn":
        return bv.knn(state["layout"])
    srv = state["server"]
    reqs = [srv.submit(j, th) for j, th in state["jobs"]]
    return [np.float64(srv.wait(r)[0]) for r in reqs]


# -------------------------------------------------------------- exact values

def _kv_scaled(x, nu):
    """x^nu K_nu(x), x > 0: the trapezoid rule on exp(-x cosh t) cosh(nu t),
    which converges geometrically (step 1/4: below 1e-17)."""
    out = torch.zeros_like(x)
    for k in range(96):
        t = 0.25 * k
        out += (0.125 if k == 0 else 0.25) * math.cosh(nu * t) * torch.exp(-x * math.cosh(t))
    return out * x ** nu


def _matern(r, sigma2, nu):
    if nu == 0.5:
        c = torch.exp(-r)
    elif nu == 1.5:
        c = (1 + r) * torch.exp(-r)
    elif nu == 2.5:
        c = (1 + r + r * r / 3) * torch.exp(-r)
    else:
        c = _kv_scaled(torch.where(r > 0, r, 1.0), nu) / (2 ** (nu - 1) * math.gamma(nu))
    return sigma2 * torch.where(r > 0, c, 1.0)


def _cov(p, case):
    """Covariance of the points p [..., m, dims]."""
    d = p[..., :, None, :] - p[..., None, :, :]
    dist = torch.sqrt((d * d).sum(-1))
    th = _theta(case)
    if not case.get("slots"):
        return _matern(dist / th[1], th[0], th[2])
    g = d[..., 2].abs() ** (2 * th[4]) / th[3] + 1
    return _matern(dist / th[1] / g ** (th[5] / 2), th[0], th[2]) / g ** (th[5] + th[6])


def _knn_sets(L, p, dev):
    """The cs nearest earlier points of every block's centroid (plane or 3-D
    distance); the order within a set does not matter to the likelihood."""
    c = np.stack([L.cx, L.cy] + ([L.cz] if L.cz is not None else []), 1)
    c = torch.as_tensor(c, device=dev)
    sets = torch.zeros((L.bc, L.cs), dtype=torch.int64, device=dev)
    step = max(1, 200_000_000 // L.n)
    acc = torch.as_tensor(L.batchNumAccum.astype(np.int64), device=dev)
    for b in range(1, L.bc, step):
        e = min(L.bc, b + step)
        lim = int(L.batchNumAccum[e - 1])
        d2 = torch.zeros((e - b, lim), dtype=torch.float64, device=dev)
        for k in range(p.shape[1]):
            d2 += (c[b:e, k:k + 1] - p[None, :lim, k]) ** 2
        d2.masked_fill_(torch.arange(lim, device=dev)[None] >= acc[b:e, None], math.inf)
        sets[b:e] = d2.topk(L.cs, dim=1, largest=False).indices
    return sets


def _exact_llk(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    L = _layout(case, seed)
    cols = [L.x, L.y] + ([L.z] if L.z is not None else [])
    p = torch.as_tensor(np.stack(cols, 1), device=dev)
    obs = torch.as_tensor(L.obs, device=dev)
    sets = _knn_sets(L, p, dev)
    acc, total = L.batchNumAccum, 0.0
    groups = {}
    for b in range(L.bc):
        groups.setdefault((int(L.batchNum[b]), b == 0), []).append(b)
    for (m, first), blocks in sorted(groups.items()):
        mc = 0 if first else L.cs
        M = mc + m
        step = max(1, 30_000_000 // (M * M))
        for s in range(0, len(blocks), step):
            bl = torch.as_tensor(blocks[s:s + step], device=dev)
            own = torch.as_tensor(acc[:-1].astype(np.int64), device=dev)[bl][:, None] + torch.arange(m, device=dev)
            pts = torch.cat([sets[bl][:, :mc], own], 1)
            C = _cov(p[pts], case)
            if case.get("nugget"):
                C = C + case["nugget"] * torch.eye(M, dtype=torch.float64, device=dev)
            F = torch.linalg.cholesky(C)
            u = torch.linalg.solve_triangular(F, obs[pts][..., None], upper=False)[:, mc:, 0]
            ld = 2 * torch.log(torch.diagonal(F, dim1=1, dim2=2)[:, mc:]).sum()
            total -= 0.5 * float((u * u).sum() + ld + len(bl) * m * math.log(2 * math.pi))
    return total


def exact(case, seed):
    kind = case["kind"]
    if kind == "knn":
        return None  # whole numbers
    if kind == "serve":
        # The jobs that take a few seconds here.
        return [np.float64(_exact_llk(c, s)) if c["n"] <= 30000 else None for c, s in _jobs(case, seed)]
    if case["nu"] == 2.5 or case["n"] * (case["cs"] + case["bs"]) ** 2 / case["bs"] > 4e9:
        return None  # failed pivots, or too long
    return np.float64(_exact_llk(case, seed))


# --------------------------------------------------------------------- work

def _eval_work(n, bs, cs):
    """Dense algebra by LAPACK's counts (potrf, trsm, gemm, potrf, trsm of one
    block's conditional density) and twelve operations per covariance entry;
    locations, observations and conditioning indices once."""
    blocks, m = n / bs, float(bs)
    potrf = lambda k: k ** 3 / 3 + k ** 2 / 2 + k / 6  # noqa: E731
    f = potrf(cs) + cs * cs * m + cs * cs + 2 * m * m * cs + 2 * m * cs + potrf(m) + m * m + 2 * m
    f += 12 * (cs + m) * (cs + m + 1) / 2
    return {"bytes": n * 24.0 + blocks * cs * 4.0, "flops": blocks * f}


def work(case):
    if case["kind"] == "knn":
        # The locations once, the sets once; one distance per selected point.
        k = case["n"] / case["bs"] * case["cs"]
        return {"bytes": case["n"] * 16.0 + 4.0 * k, "flops": 5.0 * k}
    if case["kind"] == "serve":
        ws = [_eval_work(c["n"], c["bs"], c["cs"]) for c, _ in _jobs(case, 0)]
        return {k: sum(w[k] for w in ws) for k in ("bytes", "flops")}
    return _eval_work(case["n"], case["bs"], case["cs"])
