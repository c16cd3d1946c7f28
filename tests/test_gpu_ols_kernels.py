"""run_ols against the same sums in numpy, at the sizes where its kernels can go
wrong: column counts around the blocks of 8, row counts around the steps of 16
and odd ones (no 16-byte alignment), column pointers 8 bytes off, clusters
sorted and not, empty, of one row, longer than a thread takes, and 32
consecutive ones longer than a warp stages.

FP64 sums of at most 4e4 terms in another order differ by at most n eps = 1e-11
of the sum of magnitudes; X'X of normal columns has a condition number below 10,
so 1e-10 of the largest entry bounds coefficients and covariances.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REL_TOL = 1e-10


def _reference(y, X, w, cl, G, se_type):
    n, p = X.shape
    w = np.ones(n) if w is None else w
    inv = np.linalg.inv((X * w[:, None]).T @ X)
    b = inv @ ((X * w[:, None]).T @ y)
    e = y - X @ b
    rss = float(np.sum(w * e * e))
    u2 = 0.0
    if se_type == "unadjusted":
        cov = inv * (rss / (n - p))
    elif se_type == "robust":
        Z = X * (w * e)[:, None]
        cov = inv @ (Z.T @ Z) @ inv
    else:
        S = np.zeros((G, p))
        np.add.at(S, cl, X * (w * e)[:, None])
        ncl = np.unique(cl).size
        cov = inv @ (S.T @ S) @ inv * (ncl / (ncl - 1.0)) * ((n - 1.0) / (n - p))
        u2 = float(np.sum(np.bincount(cl, weights=w * e, minlength=G) ** 2))
    return b, cov, rss, u2


def _close(a, b):
    a, b = np.asarray(a, float), np.asarray(b, float)
    return np.max(np.abs(a - b)) <= REL_TOL * max(np.max(np.abs(b)), 1e-300)


def _data(n, p, seed):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((n, p))
    return rng, X @ np.linspace(-1, 1, p) + rng.standard_normal(n), X


@pytest.mark.parametrize("se_type,weighted", [("unadjusted", False), ("robust", True), ("cluster", True)])
@pytest.mark.parametrize("p", [1, 7, 8, 9, 15, 16, 17, 23, 24, 31, 32])
@pytest.mark.parametrize("n", [48, 1001, 4096])
def test_column_and_row_counts(pkg, n, p, se_type, weighted):
    rng, y, X = _data(n, p, n + p)
    w = rng.lognormal(0.0, 0.5, n) if weighted else None
    cl = np.sort(rng.integers(0, n // 5, n)).astype(np.int32)
    _, cl = np.unique(cl, return_inverse=True)
    r = pkg.run_ols(y, X, w, cl if se_type == "cluster" else None, se_type=se_type)
    b, cov, rss, u2 = _reference(y, X, w, cl, int(cl.max()) + 1, se_type)
    assert _close(r.coefficients, b) and _close(r.covariance, cov) and _close(r.rss, rss)
    if se_type == "cluster":
        assert _close(r.cluster_u2, u2)


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n", [999, 1000])
def test_device_columns_off_a_16_byte_boundary(pkg, n, offset):
    import torch
    rng, y, X = _data(n, 13, n)
    flat = torch.zeros(14 * n + offset, dtype=torch.float64, device="cuda")
    v = flat[offset:].view(14, n)
    v[0] = torch.from_numpy(y)
    v[1:] = torch.from_numpy(np.ascontiguousarray(X.T))
    r = pkg.run_ols(v[0], v[1:], se_type="robust")
    b, cov, rss, _ = _reference(y, X, None, None, 0, "robust")
    assert _close(r.coefficients, b) and _close(r.covariance, cov) and _close(r.rss, rss)


@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("sizes", ["one", "small", "mixed", "gaps", "dense32"])
def test_cluster_sizes(pkg, sizes, shuffled):
    import torch
    rng = np.random.default_rng(7)
    count = {"one": np.ones(500, int), "small": rng.integers(1, 12, 3000),
             "mixed": np.where(rng.random(900) < 0.05, rng.integers(33, 900, 900), rng.integers(1, 33, 900)),
             "gaps": rng.integers(0, 4, 2000), "dense32": np.full(200, 32)}[sizes]
    cl = np.repeat(np.arange(count.size), count).astype(np.int32)
    if cl[-1] != count.size - 1:
        cl[-1] = count.size - 1
    n = cl.size
    _, y, X = _data(n, 5, 11)
    perm = rng.permutation(n) if shuffled else np.arange(n)
    cl = cl[perm]
    v = torch.from_numpy(np.ascontiguousarray(np.vstack([y, X.T]))).cuda()  # (columns, n), contiguous
    r = pkg.run_ols(v[0], v[1:], clusters=torch.from_numpy(cl).cuda(), se_type="cluster")
    b, cov, rss, u2 = _reference(y, X, None, cl, count.size, "cluster")
    assert r.num_clusters == np.unique(cl).size
    assert _close(r.coefficients, b) and _close(r.covariance, cov) and _close(r.cluster_u2, u2)
