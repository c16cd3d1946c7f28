"""The coefficient form of the slope solver is set up only where iterations are left
that pay for it: a solve the start satisfies, or that one check interval of
observation passes ends, makes the library calls of a panel that the form does not
take (a small dim over its limit), and a long solve those of the form.  Answers as in
the form's own tests: both forms stop once the preconditioned gradient is 1e-13 of the
column, 1e-9 of the column norm leaves room for lambda_min down to 1e-8."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solve(absorber, v, fes, G, z, opt):
    import torch
    out, r = absorber.absorb_slopes_device(torch.from_numpy(np.ascontiguousarray(v)).cuda(), [torch.from_numpy(f).cuda() for f in fes], G,
                                           [(1, torch.from_numpy(z).cuda(), True)], None, opt)
    assert r.converged
    return out.cpu().numpy(), r


def _panel(n, workers, firms, small, seed):
    rng = np.random.default_rng(seed)
    w = np.sort(rng.integers(0, workers, n)).astype(np.int32)
    return rng, [w, rng.integers(0, firms, n).astype(np.int32), rng.integers(0, small, n).astype(np.int32)], [
        workers, firms, small]


@pytest.mark.parametrize("cols,small", [(1, 8), (1, 16), (6, 36)])
def test_start_already_satisfies(absorber, pkg, cols, small):
    calls = {}
    for levels in (small, 65):
        rng, fes, G = _panel(20_000, 2_000, 90, levels, 1)
        v = rng.standard_normal((cols, G[0]))[:, fes[0]]  # in the span of the workers
        out, r = _solve(absorber, v, fes, G, rng.standard_normal(fes[0].size), pkg.make_options(tol=1e-9))
        assert r.iterations == 0 and np.all(np.abs(out) <= 1e-12 * np.abs(v).max())
        calls[levels] = r.library_calls
    assert calls[small] == calls[65]


@pytest.mark.parametrize("cols,small", [(1, 16), (6, 36)])  # 16 and 6 rounds
def test_few_iterations_and_a_long_set_up(absorber, pkg, cols, small):
    calls = {}
    for levels in (small, 65):
        rng, fes, G = _panel(60_000, 900, 10, levels, 2)
        opt = pkg.make_options(tol=1e-3, tolerance_mode=0)
        _, r = _solve(absorber, rng.standard_normal((cols, fes[0].size)), fes, G, rng.standard_normal(fes[0].size), opt)
        assert 0 < r.iterations <= 4
        calls[levels] = r.library_calls
    assert calls[small] == calls[65]


# rounds of the set-up: up to 6 it is made at once here, then after a check interval
@pytest.mark.parametrize("cols,small", [(1, 3), (1, 4), (1, 16), (2, 20), (4, 64), (6, 36), (7, 50), (13, 36)])
def test_long_solves_take_the_form(absorber, pkg, panels, cols, small):
    p = panels.akm_two_way(30_000, n_firms=400, n_years=12, seed=cols + small)  # spells at few firms: slow
    calls = {}
    for levels in (small, 65):
        rng = np.random.default_rng(cols + small)
        fes, G = [p.fes[0], p.fes[1], rng.integers(0, levels, p.n).astype(np.int32)], [*p.levels, levels]
        v, z = rng.standard_normal((cols, p.n)), rng.standard_normal(p.n)
        out, r = _solve(absorber, v, fes, G, z, pkg.make_options(tol=1e-11))
        ref, _ = _solve(absorber, v, fes, G, z, pkg.make_options(tol=1e-11, pass_kernel=1))
        assert np.all(np.linalg.norm(out - ref, axis=1) <= 1e-9 * np.linalg.norm(v, axis=1))
        assert r.iterations > 20
        calls[levels] = r.library_calls
    assert calls[small] > calls[65]
