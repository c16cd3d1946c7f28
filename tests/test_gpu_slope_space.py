"""Slopes in coefficient space (one large dimension and few small ones beside the
primary, up to 32 columns) against block Jacobi over the observations: 1 to 33
columns (tiles of 8, one and several lane slots; 33 takes the observation
passes), 0 to 65 basis columns of small dims (65 too), a primary and a large dim
with and without intercept and slope, weights, unsorted rows, empty groups,
a group of the large dim with more chunks of runs than are summed serially, and
a primary group with more runs than the form takes.

Both stop once the preconditioned gradient is 1e-13 of the column, and the
distance to the projection is at most that over sqrt(lambda_min); 1e-9 of the
column norm leaves room for lambda_min down to 1e-8.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(absorber, pkg, y, X, fes, G, slopes, w):
    v = np.column_stack([y, X])
    scale = np.linalg.norm(v, axis=0)
    out = []
    for form in (0, 1):
        r = absorber.absorb(y, X, fes, G, w, pkg.make_options(tol=1e-11, pass_kernel=form), slopes=slopes)
        assert r.converged
        out.append(np.column_stack([r.y_tilde, r.X_tilde]))
    assert np.all(np.linalg.norm(out[0] - out[1], axis=0) <= 1e-9 * scale)


def _panel(n, seed, workers, firms, small, giant=0.0):
    rng = np.random.default_rng(seed)
    f = rng.integers(0, firms, n)
    if giant:
        f[rng.random(n) < giant] = 0
    return rng, [rng.integers(0, workers, n).astype(np.int32), f.astype(np.int32)] + [
        rng.integers(0, g, n).astype(np.int32) for g in small]


@pytest.mark.parametrize("cols", [1, 2, 7, 8, 9, 13, 16, 17, 32, 33])
@pytest.mark.parametrize("small", [(), (8,)])
def test_columns(absorber, pkg, cols, small):
    n, G = 6_000, [900, 60, *small]
    rng, fes = _panel(n, cols, G[0], G[1], small)
    X = rng.standard_normal((n, cols - 1))
    _check(absorber, pkg, rng.standard_normal(n), X, fes, G, [(1, rng.standard_normal(n), True)], None)


@pytest.mark.parametrize("small", [(1,), (7,), (9, 12), (64,), (40, 25)])
@pytest.mark.parametrize("weighted", [False, True])
def test_small_dims(absorber, pkg, small, weighted):
    n, G = 8_000, [1_200, 101, *small]
    rng, fes = _panel(n, sum(small), G[0], G[1], small)
    X = rng.standard_normal((n, 5))
    w = rng.lognormal(0.0, 0.5, n) if weighted else None
    _check(absorber, pkg, rng.standard_normal(n), X, fes, G, [(1, rng.standard_normal(n), True)], w)


# (dim, with its intercept): the primary, the large and a small dim
@pytest.mark.parametrize("terms", [[], [(1, False)], [(0, True)], [(0, False), (1, False)], [(0, True), (1, True)],
                                   [(1, True), (2, True)], [(2, False)]])
def test_bases(absorber, pkg, terms):
    n, G = 9_000, [801, 72, 10]
    rng, fes = _panel(n, 5 + len(terms), 800, 70, (10,))  # groups without rows at the end of two dims
    if not any(d == 1 for d, _ in terms):
        terms = terms + [(2, True)] if not terms else terms
    slopes = [(d, rng.standard_normal(n) + 0.3, icpt) for d, icpt in terms]
    _check(absorber, pkg, rng.standard_normal(n), rng.standard_normal((n, 8)), fes, G, slopes,
           rng.lognormal(0.0, 0.3, n))


@pytest.mark.parametrize("sort", [False, True])
def test_giant_groups(absorber, pkg, sort):
    n, G = 60_000, [9_000, 500, 12]
    rng, fes = _panel(n, 3, G[0], G[1], (12,), giant=0.3)  # 18,000 rows of firm 0: over 32 chunks of runs
    if sort:
        fes[0] = np.sort(fes[0])
    slopes = [(1, rng.standard_normal(n), True)]
    y, X = rng.standard_normal(n), rng.standard_normal((n, 6))
    _check(absorber, pkg, y, X, fes, G, slopes, None)
    fes[0][rng.random(n) < 0.1] = 17  # one worker with every firm: at most 500 runs
    _check(absorber, pkg, y, X, fes, G, slopes, None)


def test_primary_group_of_many_runs(absorber, pkg):
    n, G = 40_000, [9_000, 800]
    rng, fes = _panel(n, 9, G[0], G[1], ())
    fes[0][:9_000] = 5  # 800 runs: the observation passes
    _check(absorber, pkg, rng.standard_normal(n), rng.standard_normal((n, 3)), fes, G,
           [(1, rng.standard_normal(n), True)], None)
