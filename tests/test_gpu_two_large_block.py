"""The explicit Schur block of two large dims (FP64 solves) where its build branches: rows
in any order, empty groups, a group that returns in a later run of its segment,
rows and whole segments of weight zero, segments in which one dim or the other has a
single group (it drops out there) beside segments in which both have several, the most
runs a segment may have and one more (the other form), and both orders of the dims.

Both forms stop at 1e-11 of ||b||; on these panels an error of the FE
coefficients shows up in the within transform less than a hundredfold, so 1e-9
of the column norm bounds the distance of either from the projection.  Which form
ran shows in the launches of a solve on the reused structure: the block's inner solve is
one, the pass over the observations takes several an iteration.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(absorber, pkg, oracle_mod, y, X, fes, G, w, block=True):
    v = np.column_stack([y, X])
    use = slice(None) if w is None else w > 0  # rows of weight zero have no defined transform
    scale = np.linalg.norm(v[use], axis=0)
    out, launches = [], []
    for form in (0, 1):
        o = dict(tol=1e-11, precision="fp64", pass_kernel=form)
        r = absorber.absorb(y, X, fes, G, w, pkg.make_options(**o))
        assert r.converged
        out.append(np.column_stack([r.y_tilde, r.X_tilde])[use])
        launches.append(absorber.absorb(y, X, fes, G, w, pkg.make_options(**o, reuse_structure=True)).kernel_launches)
    ref, _, ok = oracle_mod.project(y, X, fes, G, w, tol=1e-13)
    assert ok
    assert np.all(np.linalg.norm(out[0] - out[1], axis=0) <= 1e-9 * scale)
    assert np.all(np.linalg.norm(out[0] - ref[use], axis=0) <= 1e-9 * scale)
    assert launches[0] < launches[1] if block else launches[0] == launches[1]


def _columns(n, seed, cols=5):
    rng = np.random.default_rng(seed)
    return rng, rng.standard_normal(n), rng.standard_normal((n, cols - 1))


@pytest.mark.parametrize("years", [True, False])
@pytest.mark.parametrize("swap", [False, True])
def test_any_order_empty_groups_and_returning_groups(absorber, pkg, oracle_mod, panels, years, swap):
    p = panels.akm_two_way(20_000, n_firms=400, n_years=15, seed=5, three_way=True)
    rng = np.random.default_rng(2)
    spell = np.r_[True, (np.diff(p.fes[0]) != 0) | (np.diff(p.fes[1]) != 0)]
    job = rng.integers(0, 150, int(spell.sum()))[np.cumsum(spell) - 1]
    job = np.where(rng.random(p.n) < 0.1, rng.integers(0, 150, p.n), job)  # back in its group a run later
    order = rng.permutation(p.n)
    two = [p.fes[1][order], job[order].astype(np.int32)]
    lv = [int(two[0].max()) + 9, 160]
    if swap:
        two, lv = two[::-1], lv[::-1]
    fes, G = [p.fes[0][order], *two], [int(p.fes[0].max()) + 4, *lv]
    if years:
        fes, G = fes + [p.fes[2][order]], G + [int(p.fes[2].max()) + 3]
    w = rng.lognormal(0.0, 0.5, p.n)
    w[rng.random(p.n) < 0.02] = 0.0
    w[np.isin(fes[0], rng.integers(0, G[0], 20))] = 0.0  # whole segments
    _check(absorber, pkg, oracle_mod, p.y[order], p.X[order], fes, G, w)


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("years", [True, False])
def test_dims_of_one_group_in_a_segment(absorber, pkg, oracle_mod, weighted, years):
    n = 24_000
    rng, y, X = _columns(n, 6)
    worker = np.repeat(np.arange(n // 8), 8).astype(np.int32)
    firm, job = rng.integers(0, 300, n), rng.integers(0, 200, n)
    kind = rng.integers(0, 4, n // 8)[worker]  # 0 both several, 1 one firm, 2 one job, 3 one of each
    first = worker * 8
    firm = np.where((kind == 1) | (kind == 3), firm[first], firm)
    job = np.where((kind == 2) | (kind == 3), job[first], job)
    # of the others, two groups each in runs of two and three
    half = np.arange(n) % 8
    firm = np.where(kind == 0, firm[first + (half // 2) * 2 % 4], firm)
    job = np.where(kind == 0, job[first + (half // 3) % 2], job)
    firm = np.where(kind == 2, firm[first + half // 4], firm)
    job = np.where(kind == 1, job[first + half // 4], job)
    fes, G = [worker, firm.astype(np.int32), job.astype(np.int32)], [n // 8, 300, 200]
    if years:
        fes, G = fes + [rng.integers(0, 12, n).astype(np.int32)], G + [12]
    _check(absorber, pkg, oracle_mod, y, X, fes, G, rng.lognormal(0.0, 0.5, n) if weighted else None)


@pytest.mark.parametrize("runs,block", [(64, True), (65, False)])
def test_most_runs_of_a_segment(absorber, pkg, oracle_mod, runs, block):
    # one worker with `runs` runs of both dims together, the others with few
    n = 16_000
    rng, y, X = _columns(n, 7)
    worker = 1 + np.arange(n) // 4
    firm = rng.integers(0, 120, n // 2)[np.arange(n) // 2]
    job = rng.integers(0, 90, n // 4 + 1)[worker - 1]
    lead = 96
    worker[:lead] = 0
    f_runs, j_runs = runs - 24, 24
    firm[:lead] = np.minimum(np.arange(lead) * f_runs // lead, f_runs - 1)
    job[:lead] = np.minimum(np.arange(lead) * j_runs // lead, j_runs - 1)
    worker = np.unique(worker, return_inverse=True)[1]
    fes = [worker.astype(np.int32), firm.astype(np.int32), job.astype(np.int32)]
    assert sum(1 + int((np.diff(f[:lead]) != 0).sum()) for f in fes[1:]) == runs
    G = [int(worker.max()) + 1, 120, 90]
    _check(absorber, pkg, oracle_mod, y, X, fes, G, None, block)
