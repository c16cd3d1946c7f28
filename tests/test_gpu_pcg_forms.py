"""The persistent PCG over the explicit Schur block against the run-level matvec
and the oracle: one cluster and the whole grid, 4, 8 and 16 columns, no small
dim and small dims of few, many and the most levels a lane holds, rows of every
length (empty, short, several chunks, more chunks than one lane group sums),
FP32 inside FP64 refinement and FP64 throughout.

Both forms stop at 1e-11 of ||b||; on these panels an error of the FE
coefficients shows up in the within transform less than a hundredfold, so 1e-9
of the column norm bounds the distance of either from the projection.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _columns(absorber, pkg, p, fes, G, cols, precision, form, seed):
    rng = np.random.default_rng(seed)
    X = np.column_stack([p.X, rng.standard_normal((p.n, max(cols - 3, 0)))])[:, : cols - 1]
    o = pkg.make_options(tol=1e-11, precision=precision, pass_kernel=form)
    r = absorber.absorb(p.y, X, fes, G, p.weights, o)
    assert r.converged
    return np.column_stack([p.y, X]), np.column_stack([r.y_tilde, r.X_tilde])


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("cols,years", [(1, 0), (3, 10), (5, 33), (7, 0), (9, 40), (13, 41), (16, 64), (11, 2)])
@pytest.mark.parametrize("n,firms", [(2_000, 40), (30_000, 900)])
def test_persistent_pcg_equals_run_level(absorber, pkg, oracle_mod, panels, n, firms, cols, years, precision):
    p = panels.akm_two_way(n, n_firms=firms, n_years=max(years, 12), seed=cols + years, three_way=years > 0)
    rng = np.random.default_rng(5)
    p.weights = rng.lognormal(0.0, 0.5, p.n) if cols % 2 else None
    fes, G = p.fes, p.levels
    if years > 0:  # any number of levels: the years folded or spread over `years` levels
        t = (p.fes[2] + (np.arange(p.n) % 7) * 12) % years
        t[:years] = np.arange(years)
        fes, G = [p.fes[0], p.fes[1], t.astype(np.int32)], [p.levels[0], p.levels[1], years]
    v, a = _columns(absorber, pkg, p, fes, G, cols, precision, 0, 3)
    _, b = _columns(absorber, pkg, p, fes, G, cols, precision, 3, 3)
    scale = np.linalg.norm(v, axis=0)
    assert np.all(np.linalg.norm(a - b, axis=0) <= 1e-9 * scale)
    ref, _, ok = oracle_mod.project(v[:, 0], v[:, 1:], fes, G, p.weights, tol=1e-13)
    assert ok and np.all(np.linalg.norm(a - ref, axis=0) <= 1e-9 * scale)


@pytest.mark.parametrize("cols,precision", [(3, "mixed"), (13, "mixed"), (4, "fp64")])
def test_rows_of_many_chunks(absorber, pkg, panels, cols, precision):
    # one firm linked to almost every other one: its row has over 16 chunks of 256
    p = panels.akm_two_way(150_000, n_firms=6_000, seed=3, three_way=True, zipf=0.3, move_prob=0.3)
    f = p.fes[1].copy()
    f[np.flatnonzero(np.arange(p.n) % 4 == 0)] = 0
    f, gf = pkg.dense_ids(f)
    fes, G = [p.fes[0], f, p.fes[2]], [p.levels[0], gf, p.levels[2]]
    v, a = _columns(absorber, pkg, p, fes, G, cols, precision, 0, 3)
    _, b = _columns(absorber, pkg, p, fes, G, cols, precision, 3, 3)
    assert np.all(np.linalg.norm(a - b, axis=0) <= 1e-9 * np.linalg.norm(v, axis=0))
