"""Two large dims beside the primary (worker, firm, year, occupation and the
like): the explicit Schur block (solves in FP64 throughout) and the pass over the
observations (mixed), against the observation-level form and the oracle: with and without a coupled small dim, weights, unsorted rows, empty
groups, workers in one firm or one occupation only, groups met again later in a
segment, more runs in a segment than the explicit block takes (the other form),
4 to 16 columns and both precisions.

Both forms stop at 1e-11 of ||b||; on these panels an error of the FE
coefficients shows up in the within transform less than a hundredfold, so 1e-9
of the column norm bounds the distance of either from the projection.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _panel(panels, n, firms, jobs, seed, extra=0.0):
    p = panels.akm_two_way(n, n_firms=firms, n_years=15, seed=seed, three_way=True)
    rng = np.random.default_rng(seed)
    spell = np.flatnonzero(np.r_[True, (np.diff(p.fes[0]) != 0) | (np.diff(p.fes[1]) != 0) | (rng.random(p.n - 1) < extra)])
    job = np.zeros(p.n, np.int64)
    job[spell] = rng.integers(0, jobs, spell.size)
    idx = np.zeros(p.n, np.int64)
    idx[spell] = spell
    job = job[np.maximum.accumulate(idx)]
    return p, np.unique(job, return_inverse=True)[1].astype(np.int32)


def _check(absorber, pkg, oracle_mod, y, X, fes, G, w, precision="mixed"):
    v = np.column_stack([y, X])
    scale = np.linalg.norm(v, axis=0)
    out = []
    for form in (0, 1):
        r = absorber.absorb(y, X, fes, G, w, pkg.make_options(tol=1e-11, precision=precision, pass_kernel=form))
        assert r.converged
        out.append(np.column_stack([r.y_tilde, r.X_tilde]))
    ref, _, ok = oracle_mod.project(y, X, fes, G, w, tol=1e-13)
    assert ok
    assert np.all(np.linalg.norm(out[0] - out[1], axis=0) <= 1e-9 * scale)
    assert np.all(np.linalg.norm(out[0] - ref, axis=0) <= 1e-9 * scale)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("n,firms,jobs,years,weighted,cols", [
    (2_000, 70, 66, True, False, 1), (2_000, 70, 80, False, True, 3), (30_000, 900, 120, True, True, 7),
    (30_000, 300, 2_000, True, False, 16), (30_000, 900, 120, False, False, 13)])
def test_explicit_block_of_two_large_dims(absorber, pkg, oracle_mod, panels, n, firms, jobs, years, weighted, cols,
                                          precision):
    p, job = _panel(panels, n, firms, jobs, seed=n + jobs, extra=0.05)
    rng = np.random.default_rng(1)
    X = np.column_stack([p.X, rng.standard_normal((p.n, max(cols - 3, 0)))])[:, : cols - 1]
    fes = [p.fes[0], p.fes[1], p.fes[2], job] if years else [p.fes[0], p.fes[1], job]
    G = [int(f.max()) + 1 for f in fes]
    w = rng.lognormal(0.0, 0.5, p.n) if weighted else None
    _check(absorber, pkg, oracle_mod, p.y, X, fes, G, w, precision)


def test_unsorted_rows_empty_groups_and_regrouped_runs(absorber, pkg, oracle_mod, panels):
    p, job = _panel(panels, 20_000, 400, 150, seed=5, extra=0.1)
    rng = np.random.default_rng(2)
    back = rng.random(p.n) < 0.1  # single rows of another occupation: a group returns in a later run
    job = np.where(back, rng.integers(0, 150, p.n), job).astype(np.int32)
    order = rng.permutation(p.n)
    fes = [p.fes[0][order], job[order], p.fes[2][order], p.fes[1][order]]
    G = [int(fes[0].max()) + 4, 160, int(fes[2].max()) + 1, int(fes[3].max()) + 9]
    w = rng.lognormal(0.0, 0.5, p.n)
    w[:50] = 0.0
    _check(absorber, pkg, oracle_mod, p.y[order], p.X[order], fes, G, w)


def test_long_segments_keep_the_other_form(absorber, pkg, oracle_mod, panels):
    p, job = _panel(panels, 12_000, 300, 100, seed=9)
    rng = np.random.default_rng(3)
    worker = np.sort(rng.integers(0, 500, p.n)).astype(np.int32)
    firm = rng.integers(0, 400, p.n).astype(np.int32)
    worker[:90] = 0  # over 64 runs in one segment
    G = [int(worker.max()) + 1, 400, int(job.max()) + 1, int(p.fes[2].max()) + 1]
    _check(absorber, pkg, oracle_mod, p.y, p.X, [worker, firm, job, p.fes[2]], G, None)
