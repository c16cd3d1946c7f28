"""The absorber's performance cases: what a user's program has it do, through the package's entry points.

Panels are the seeded worker-firm-year designs of ``panels.py`` (spells of 1 + Poisson(9) years, Zipf firms,
10% moves a year), made here on the GPU from the seed alone.  They hold no singletons by construction (workers
have two rows or more, a firm seen once joins the largest one), so that a case has its n rows for every seed:

* ``basic``  -- y, x1, x2 with worker, firm and year effects (the plain two-way design);
* ``spells`` -- y, tenure, tenure^2, age, age^2, age^3 and normal controls (the 50M three-way design).

``tol`` is the absorption's own stopping rule: 1e-10 for whoever needs coefficients and standard errors to 1e-8 of
a CPU fit, as the repository's parity tests do; 1e-8, the library's default, for the headline and panels near it.
"""

from __future__ import annotations

import math
import time

import numpy as np
import torch

import __graft_entry__ as ge

pkg = ge.load_package()

DEVICE = "cuda:0"
EXACT_SECONDS = 18.0  # exact() gives up on a case that takes longer

ABSORB = {"kind": "absorb", "design": "basic", "firms_per": 60, "years": 20, "dims": 3, "controls": 0,
          "weighted": False, "shuffled": False, "precision": "mixed", "tol": 1e-10}


def listed():
    def absorb(name, n, **kw):
        return {**ABSORB, "name": name, "n": n, **kw}

    return [
        # One small panel of a batch of independent fits (the smallest sizes of the uneven batch):
        # launches, synchronisations and grid-wide barriers are all there is.
        absorb("absorb_10k_2way_3col", 10_000, dims=2),
        # A mid-sized weighted panel of the same batch, odd number of rows, three FE dims.
        absorb("absorb_300k_3way_weighted", 300_007, weighted=True),
        # The plain design at its stated size: 1M rows, 10 years, 10k firms, outcome and two regressors, rows
        # as a data base hands them over (not in worker order).
        absorb("absorb_1M_2way_unsorted", 1_000_000, dims=2, firms_per=100, years=10, shuffled=True),
        # The same size as a wage regression: outcome and 12 regressors, three FE dims, solved throughout in
        # 64 bits, the caller's choice where the inputs are badly scaled.
        absorb("absorb_1M_3way_13col_fp64", 1_000_000, design="spells", controls=7, years=36, precision="fp64"),
        # Worker, firm, year and occupation: a second large dim beside the firms, as in the four-way panels that
        # the parity tests and the warm start's workload have; ragged size and columns.
        absorb("absorb_2M_4way_9col", 2_000_003, design="spells", controls=3, dims=4, years=36),
        # The headline workload's shape at a tenth of its rows, with analytic weights.
        absorb("absorb_5M_3way_13col_weighted", 5_000_000, design="spells", controls=7, years=36, weighted=True),
        # The headline workload: 50M rows, 800k firms, 36 years, outcome and 12 regressors.
        absorb("absorb_50M_3way_13col", 50_000_000, design="spells", controls=7, years=36, firms_per=62, tol=1e-8),
        # Host arrays in, host arrays out: how the R, Stata and Python front ends call the absorber.
        {**ABSORB, "kind": "host", "name": "host_2M_3way_8col", "n": 2_000_000, "design": "spells", "controls": 2,
         "years": 36},
        # Firm-specific tenure slopes (worker + firm##c.tenure + year).
        {**ABSORB, "kind": "slopes", "name": "slopes_4M_13col", "n": 4_000_000, "design": "spells", "controls": 7,
         "years": 36},
        # The regression after an absorption: 12 regressors, standard errors clustered by worker.
        {"kind": "ols", "name": "ols_10M_12reg_cluster", "n": 10_000_000, "p": 12, "se_type": "cluster",
         "weighted": False},
        # The leave-out firm system of a 4M-row panel, one full batch of 64 right-hand sides, host arrays.
        {"kind": "kss", "name": "kss_4M_64rhs", "n": 4_000_000, "rhs": 64},
        # Preparing a 20M-row panel: dense ids of three raw columns, singleton cascade (one row in 500 has an
        # employer of its own), mobility groups.
        {"kind": "prep", "name": "prep_20M", "n": 20_000_000, "years": 36, "firms_per": 62},
    ]


def draw(rng):
    def size(lo, hi):
        return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))

    kind = rng.choice(["absorb"] * 7 + ["host", "slopes", "ols", "kss", "prep"])
    if kind in ("absorb", "host", "slopes"):
        top = {"absorb": 30_000_000, "host": 4_000_000, "slopes": 8_000_000}[kind]
        design = "spells" if kind == "slopes" else rng.choice(["basic", "spells"])
        dims = 3 if kind == "slopes" else rng.choice([2, 3, 3, 4])
        n = size(8_000, min(top, 4_000_000) if dims == 4 else top)
        return {**ABSORB, "kind": kind, "n": n, "design": design, "dims": dims,
                "firms_per": rng.choice([40, 60, 62, 80, 100]), "years": rng.choice([10, 20, 36]),
                "controls": rng.randint(0, 7) if design == "spells" else 0,
                "weighted": kind != "slopes" and rng.random() < 0.4, "shuffled": rng.random() < 0.25,
                "tol": 1e-8 if n > 10_000_000 else 1e-10,
                "precision": "fp64" if rng.random() < 0.15 and kind == "absorb" else "mixed"}
    if kind == "ols":
        return {"kind": "ols", "n": size(50_000, 20_000_000), "p": rng.randint(1, 20),
                "se_type": rng.choice(["cluster", "cluster", "robust", "unadjusted"]),
                "weighted": rng.random() < 0.4}
    if kind == "kss":
        return {"kind": "kss", "n": size(100_000, 6_000_000), "rhs": rng.randint(1, 64)}
    return {"kind": "prep", "n": size(50_000, 30_000_000), "years": rng.choice([10, 20, 36]),
            "firms_per": rng.choice([40, 62, 100])}


# ---------------------------------------------------------------------------
# panels
# ---------------------------------------------------------------------------
def _dense(ids):
    present = torch.bincount(ids) > 0
    return (torch.cumsum(present, 0) - 1)[ids], int(present.sum())


def _spells(n, firms, years, gen, move=0.1, zipf=1.1):
    """Worker, firm, year, tenure (int64) of n rows in worker order."""
    rand = lambda m: torch.rand(m, generator=gen, device=DEVICE, dtype=torch.float64)  # noqa: E731
    mean = min(10, years)
    count = int(n / mean * 1.3) + 64
    T = torch.poisson(torch.full((count,), 9.0, device=DEVICE), generator=gen).long().add_(1).clamp_(2, years)
    while int(T.sum()) < n:
        T = torch.cat([T, T])
    cum = torch.cumsum(T, 0)
    W = int(torch.searchsorted(cum, n)) + 1
    T = T[:W].clone()
    T[-1] -= int(cum[W - 1]) - n
    if int(T[-1]) == 1:  # no worker with a single row
        T[-1] += 1
        T[T.argmax()] -= 1
    start = (rand(W) * (years - T + 1)).long()
    worker = torch.repeat_interleave(torch.arange(W, device=DEVICE), T, output_size=n)
    rows = torch.arange(n, device=DEVICE)
    pos = rows - (torch.cumsum(T, 0) - T)[worker]
    begin = (pos == 0) | (rand(n) < move)
    cdf = torch.cumsum(torch.arange(1, firms + 1, device=DEVICE, dtype=torch.float64) ** -zipf, 0)
    ids = torch.randperm(firms, generator=gen, device=DEVICE)
    firm = torch.zeros(n, dtype=torch.int64, device=DEVICE)
    m = int(begin.sum())
    firm[begin] = ids[torch.searchsorted(cdf / cdf[-1], rand(m), right=True).clamp_(max=firms - 1)]
    first = torch.cummax(torch.where(begin, rows, 0), 0).values
    firm = firm[first]
    firm = torch.where(torch.bincount(firm)[firm] > 1, firm, ids[0])  # firms seen once join the largest
    return worker, firm, start[worker] + pos, rows - first, pos


def _panel(case, seed):
    """The case's panel on the GPU: v (columns, n), int32 ids and levels of its FE dims, weights, tenure."""
    gen = torch.Generator(DEVICE).manual_seed(int(seed) * 7919 + 11)
    norm = lambda m: torch.randn(m, generator=gen, device=DEVICE, dtype=torch.float64)  # noqa: E731
    firms = max(100, case["n"] // case["firms_per"])
    w, f, t, ten, pos = _spells(case["n"], firms, case["years"], gen)
    W = int(w[-1]) + 1
    fe_w, fe_f, fe_t = norm(W), 0.5 * norm(firms), 0.1 * norm(case["years"])
    age0 = torch.randint(20, 46, (W,), generator=gen, device=DEVICE).double()
    n = case["n"]
    if case["shuffled"]:
        rows = torch.randperm(n, generator=gen, device=DEVICE)
        w, f, t, ten, pos = (a[rows] for a in (w, f, t, ten, pos))
    effect = fe_w[w] + fe_f[f] + fe_t[t]
    if case["design"] == "basic":
        v = torch.empty(3, n, device=DEVICE, dtype=torch.float64)
        for c in (1, 2):
            v[c] = 0.3 * fe_w[w] + math.sqrt(0.91) * norm(n)
        v[0] = 0.5 * v[1] - 0.3 * v[2] + effect + norm(n)
    else:
        v = torch.empty(6 + case["controls"], n, device=DEVICE, dtype=torch.float64)
        v[1], v[2], v[3] = ten, ten * ten, age0[w] + pos
        v[4] = v[3] * v[3]
        v[5] = v[4] * v[3]
        v[0] = effect + 0.02 * v[1] - 0.0005 * v[2] + 0.01 * v[3] + norm(n)
        for c in range(6, v.shape[0]):
            v[c] = norm(n)
            v[0] += 0.1 * v[c]
    dims = [w, f, t][: case["dims"]]
    if case["dims"] >= 4:  # occupation: drawn anew at every change of employer
        jobs = max(100, firms // 20)
        drawn = torch.randint(0, jobs, (n,), generator=gen, device=DEVICE)
        spell = w * case["years"] + t - ten  # the worker and the year in which the spell began
        dims.append(drawn[spell % n])
    ids, levels = [], []
    for g in dims:
        d, G = _dense(g)
        ids.append(d.int())
        levels.append(G)
    weights = torch.exp(0.5 * norm(n)) if case["weighted"] else None
    return {"v": v, "ids": ids, "levels": levels, "weights": weights, "tenure": ten.double()}


def _components(a, b, na, nb):
    """Smallest node label of each node's component in the bipartite graph of the edges (a, na + b)."""
    label = torch.arange(na + nb, device=DEVICE)
    b = b + na
    while True:
        old = label.clone()
        low = torch.minimum(label[a], label[b])
        label.scatter_reduce_(0, a, low, "amin")
        label.scatter_reduce_(0, b, low, "amin")
        label = label[label]
        if torch.equal(label, old):
            return label


def _matches(case, seed):
    """Worker-firm matches of one mobility group, sorted by worker, with their person-years."""
    gen = torch.Generator(DEVICE).manual_seed(int(seed) * 7919 + 12)
    firms = max(1000, case["n"] // 100)
    w, f, _, _, _ = _spells(case["n"], firms, 10, gen, move=0.15)
    # one more match of every firm with a worker of the largest firm: all firms are in one mobility group
    hub = w[f == torch.bincount(f).argmax()]
    w = torch.cat([w, hub[torch.randint(0, hub.numel(), (firms,), generator=gen, device=DEVICE)]])
    f = torch.cat([f, torch.arange(firms, device=DEVICE)])
    key, count = torch.unique(w * firms + f, return_counts=True)
    return (key // firms, int(w.max()) + 1), (key % firms, firms), count.double()


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
_context = []


def _absorber():
    """One absorber context for all panels, as a program that fits many of them keeps it."""
    if not _context:
        _context.append(pkg.Absorber(0))
    return _context[0]


def _ols_inputs(case, seed):
    """Within-transformed looking columns (p regressors and an outcome with cluster effects) and worker ids."""
    gen = torch.Generator(DEVICE).manual_seed(int(seed) * 7919 + 13)
    n, p = case["n"], case["p"]
    worker = _spells(n, max(100, n // 60), 36, gen)[0]
    X = torch.randn(p, n, generator=gen, device=DEVICE, dtype=torch.float64)
    beta = torch.linspace(-0.5, 0.5, p, device=DEVICE, dtype=torch.float64)
    shared = torch.randn(int(worker[-1]) + 1, generator=gen, device=DEVICE, dtype=torch.float64)
    y = torch.randn(n, generator=gen, device=DEVICE, dtype=torch.float64) + 0.3 * shared[worker]
    X[0] += 0.2 * shared[worker]
    for j in range(p):
        y += beta[j] * X[j]
    weights = torch.exp(0.5 * torch.randn(n, generator=gen, device=DEVICE, dtype=torch.float64))
    return y, X, worker.int(), weights if case["weighted"] else None


def _raw_ids(case, seed):
    """Raw worker, firm and year columns: ids spread over a sparse range, with singletons."""
    gen = torch.Generator(DEVICE).manual_seed(int(seed) * 7919 + 14)
    n = case["n"]
    w, f, t, _, _ = _spells(n, max(100, n // case["firms_per"]), case["years"], gen)
    alone = torch.randperm(n, generator=gen, device=DEVICE)[: n // 500]
    f[alone] = int(f.max()) + 1 + torch.arange(n // 500, device=DEVICE)
    return [(g * 7 + 3).int() for g in (w, f, t)]


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind in ("absorb", "host", "slopes"):
        p = _panel(case, seed)
        s["options"] = pkg.make_options(tol=case["tol"], precision=case["precision"])
        s["absorber"] = _absorber()
        if kind == "host":
            host = p["v"].cpu().numpy()
            s |= {"y": host[0].copy(), "X": host[1:].copy().T, "ids": [g.cpu().numpy() for g in p["ids"]],
                  "levels": p["levels"], "weights": None if p["weights"] is None else p["weights"].cpu().numpy()}
        else:
            s |= p
            s["out"] = torch.empty_like(p["v"])
    elif kind == "ols":
        s["y"], s["X"], s["clusters"], s["weights"] = _ols_inputs(case, seed)
    elif kind == "kss":
        (w, N), (f, J), count = _matches(case, seed)
        s["solver"] = pkg.KssSolver(pkg.kss_system(w.cpu().numpy(), f.cpu().numpy(), count.cpu().numpy(), N, J))
        s["rhs"] = np.random.default_rng(int(seed)).standard_normal((case["rhs"], J))
    else:
        s["raw"] = _raw_ids(case, seed)
    return s


def run(s):
    kind = s["kind"]
    if kind == "absorb":
        out, r = s["absorber"].absorb_device(s["v"], s["ids"], s["levels"], s["weights"], s["options"], out=s["out"],
                                             stream=torch.cuda.current_stream().cuda_stream)
        return {"v": out, "converged": bool(r.converged)}
    if kind == "host":
        r = s["absorber"].absorb(s["y"], s["X"], s["ids"], s["levels"], s["weights"], s["options"])
        return {"y": r.y_tilde, "X": r.X_tilde, "converged": r.converged}
    if kind == "slopes":
        out, r = s["absorber"].absorb_slopes_device(s["v"], s["ids"], s["levels"], [(1, s["tenure"], True)], s["weights"],
                                                    s["options"], out=s["out"],
                                                    stream=torch.cuda.current_stream().cuda_stream)
        return {"v": out, "converged": bool(r.converged)}
    if kind == "ols":
        cl = s["clusters"] if s["case"]["se_type"] == "cluster" else None
        r = pkg.run_ols(s["y"], s["X"], s["weights"], cl, se_type=s["case"]["se_type"])
        return {"coefficients": r.coefficients, "covariance": r.covariance, "std_errors": r.std_errors,
                "xtx_inv": r.xtx_inv, "rss": r.rss, "clusters": r.num_clusters}
    if kind == "kss":
        z, its = s["solver"].solve_multi(s["rhs"], tol=1e-10, max_iter=20_000)
        return {"z": z, "converged": its >= 0}
    dense = [pkg.dense_ids_device(r) for r in s["raw"]]
    ids, levels = [d for d, _, _ in dense], [g for _, g, _ in dense]
    keep, dropped, rounds = pkg.drop_singletons_device(ids, levels)
    c = pkg.first_pair_component_stats(ids[0], ids[1])
    return {"ids": ids, "levels": levels, "keep": keep, "dropped": dropped, "rounds": rounds,
            "components": c.num_components, "largest": c.largest_component_n_obs,
            "share": c.largest_component_obs_share}


def work(case):
    """Inputs read once, outputs written once; operations of the sums that the result cannot do without."""
    n, kind = case["n"], case["kind"]
    if kind in ("absorb", "host", "slopes"):
        cols = 3 if case["design"] == "basic" else 6 + case["controls"]
        extra = 8 * case["weighted"] + 8 * (kind == "slopes")
        return {"bytes": n * (16.0 * cols + 4 * case["dims"] + extra), "flops": 2.0 * n * cols * case["dims"]}
    if kind == "ols":
        cols = case["p"] + 1
        return {"bytes": n * (8.0 * cols + 4 * (case["se_type"] == "cluster") + 8 * case["weighted"]),
                "flops": n * cols * (cols + 1.0)}
    if kind == "kss":
        # matches (about 0.24 a row): ids and weight; right-hand sides in, solutions out
        return {"bytes": 0.24 * n * 16.0 + 16.0 * case["rhs"] * n / 100, "flops": 4.0 * 0.24 * n * case["rhs"]}
    return {"bytes": n * (3 * 8.0 + 1), "flops": 0.0}


# ---------------------------------------------------------------------------
# the same results in 64 bits, in plain torch
# ---------------------------------------------------------------------------
class _Basis:
    """Orthonormal columns of one FE block: entry u of row i in group g[i]; D'x and D a."""

    def __init__(self, g, G, u):
        norm = torch.zeros(G, device=DEVICE, dtype=torch.float64).index_add_(0, g, u * u)
        inv = torch.where(norm > 1e-12 * norm.max(), norm.clamp(min=1e-300).rsqrt(), torch.zeros_like(norm))
        self.g, self.u = g, u * inv[g]
        order = torch.argsort(g, stable=True)
        ptr = torch.zeros(G + 1, dtype=torch.int64, device=DEVICE)
        ptr[1:] = torch.cumsum(torch.bincount(g, minlength=G), 0)
        self.t = torch.sparse_csr_tensor(ptr, order, self.u[order], (G, g.numel()))

    def down(self, x):
        return self.t @ x

    def up(self, a):
        return a[self.g] * self.u[:, None]


def _project(v, ids, levels, weights, tenure=None):
    """v (columns, n) without the span of the FEs (of firm##c.tenure too): CGLS after the first dim's exact removal."""
    began = time.monotonic()
    n = v.shape[1]
    root = torch.ones(n, device=DEVICE, dtype=torch.float64) if weights is None else weights.sqrt()
    ids = [g.long() for g in ids]
    first = _Basis(ids[0], levels[0], root)
    blocks = [_Basis(g, G, root) for g, G in zip(ids[1:], levels[1:])]
    if tenure is not None:
        z = tenure * root
        blocks.append(_Basis(ids[1], levels[1], z - blocks[0].up(blocks[0].down(z[:, None]))[:, 0]))
    off = lambda x: x - first.up(first.down(x))  # noqa: E731
    r = off(off((v * root).T.contiguous()))
    scale = (v * root).square().sum(1)
    for _ in range(2):  # started again once from its own result
        s = [b.down(r) for b in blocks]
        p = [x.clone() for x in s]
        gamma = sum(x.square().sum(0) for x in s)
        least, since = gamma.clone(), 0
        for _ in range(4000):
            if bool((gamma <= 1e-28 * scale).all()) or since > 60:
                break
            if time.monotonic() - began > EXACT_SECONDS:
                return None
            q = off(sum(b.up(x) for b, x in zip(blocks, p)))
            qq = q.square().sum(0)
            alpha = torch.where(gamma > 1e-30 * scale, gamma / qq.clamp(min=1e-300), torch.zeros_like(gamma))
            r -= alpha * q
            s = [b.down(r) for b in blocks]
            new = sum(x.square().sum(0) for x in s)
            beta = torch.where(alpha > 0, new / gamma.clamp(min=1e-300), torch.zeros_like(gamma))
            p = [x + beta * y for x, y in zip(s, p)]
            gamma = new
            since = 0 if bool((gamma < 0.5 * least).any()) else since + 1
            least = torch.minimum(least, gamma)
        r = off(r)
    return (r.T / root).contiguous()


def _exact_ols(case, seed):
    y, X, g, w = _ols_inputs(case, seed)
    n, p = y.numel(), X.shape[0]
    w = torch.ones_like(y) if w is None else w
    xtx = (X * w) @ X.T
    inv = torch.linalg.inv(xtx)
    b = inv @ (X @ (w * y))
    e = y - X.T @ b
    rss = float((w * e * e).sum())
    G = 0
    if case["se_type"] == "unadjusted":
        cov = inv * (rss / (n - p))
    elif case["se_type"] == "robust":
        cov = inv @ ((X * (w * e) ** 2) @ X.T) @ inv
    else:
        G = int(g.max()) + 1
        S = torch.zeros(G, p, device=DEVICE, dtype=torch.float64).index_add_(0, g.long(), (X * (w * e)).T)
        cov = G / (G - 1) * (n - 1) / (n - p) * inv @ (S.T @ S) @ inv
    out = [t.cpu().numpy() for t in (b, cov, cov.diagonal().sqrt(), inv)]
    return {"coefficients": out[0], "covariance": out[1], "std_errors": out[2], "xtx_inv": out[3], "rss": rss,
            "clusters": None}


def _exact_kss(case, seed):
    (w, N), (f, J), c = _matches(case, seed)
    b = torch.from_numpy(np.random.default_rng(int(seed)).standard_normal((case["rhs"], J))).to(DEVICE).T.contiguous()
    b[J - 1] = 0
    Dw = torch.zeros(N, device=DEVICE, dtype=torch.float64).index_add_(0, w, c)
    Df = torch.zeros(J, device=DEVICE, dtype=torch.float64).index_add_(0, f, c)
    diag = Df - torch.zeros_like(Df).index_add_(0, f, c * c / Dw[w])
    half = c / Dw[w].sqrt()

    def csr(rows, cols, R, C):
        order = torch.argsort(rows * C + cols)
        ptr = torch.zeros(R + 1, dtype=torch.int64, device=DEVICE)
        ptr[1:] = torch.cumsum(torch.bincount(rows, minlength=R), 0)
        return torch.sparse_csr_tensor(ptr, cols[order], half[order], (R, C))

    B, Bt = csr(w, f, N, J), csr(f, w, J, N)

    def apply(x):
        y = Df[:, None] * x - Bt @ (B @ x)
        y[J - 1] = 0
        return y

    began = time.monotonic()
    z = torch.zeros_like(b)
    inv = torch.where(diag > 0, 1 / diag, torch.zeros_like(diag))[:, None]
    scale = b.square().sum(0)
    for _ in range(3):  # refined from its own residual
        r = b - apply(z)
        r[J - 1] = 0
        p = q = inv * r
        rho = (r * q).sum(0)
        for _ in range(4000):
            if bool((r.square().sum(0) <= 1e-26 * scale).all()):
                break
            if time.monotonic() - began > EXACT_SECONDS:
                return None
            a = apply(p)
            alpha = torch.where(rho > 0, rho / (p * a).sum(0).clamp(min=1e-300), torch.zeros_like(rho))
            z += alpha * p
            r -= alpha * a
            q = inv * r
            new = (r * q).sum(0)
            p = q + new / rho.clamp(min=1e-300) * p
            rho = new
    return {"z": z.T.contiguous(), "converged": None}


def _exact_prep(case, seed):
    w, f = (_dense(g.long()) for g in _raw_ids(case, seed)[:2])
    label = _components(w[0], f[0], w[1], f[1])[w[0]]
    return {"ids": None, "levels": None, "keep": None, "dropped": None, "rounds": None, "components": None,
            "largest": None, "share": float(torch.bincount(label).max()) / case["n"]}


def exact(case, seed):
    kind = case["kind"]
    if kind == "ols":
        return _exact_ols(case, seed)
    if kind == "kss":
        return _exact_kss(case, seed)
    if kind == "prep":
        return _exact_prep(case, seed)
    p = _panel(case, seed)
    v = _project(p["v"], p["ids"], p["levels"], p["weights"], p["tenure"] if kind == "slopes" else None)
    if v is None:
        return None
    if kind == "host":
        v = v.cpu().numpy()
        return {"y": v[0], "X": v[1:].T, "converged": None}
    return {"v": v, "converged": None}
