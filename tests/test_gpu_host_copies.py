"""Host arrays in pageable memory go through the copy workers, pinned ones are
copied directly: the same bytes come back, for columns under and over the size
from which the workers run, one and several column groups, ragged last pieces,
weights, saved coefficients, and results written over the inputs."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pinned(a):
    import torch
    t = torch.empty(a.size, dtype=torch.from_numpy(a[:0].copy()).dtype, pin_memory=True).numpy()
    v = t.reshape(a.shape, order="F")
    v[...] = a
    return v


@pytest.mark.parametrize("n,cols,weighted,save", [
    (131_072, 7, False, False),   # just under the least size
    (131_072, 8, True, False),    # at it: whole pieces
    (300_001, 4, False, True), (300_001, 9, True, False), (1_100_003, 1, False, False), (1_100_003, 13, True, True)])
def test_pageable_and_pinned_arrays(absorber, pkg, n, cols, weighted, save):
    rng = np.random.default_rng(n + cols)
    G = [n // 8 + 1, n // 50 + 1, 12]
    fes = [rng.integers(0, g, n).astype(np.int32) for g in G]
    y = rng.standard_normal(n)
    X = np.asfortranarray(rng.standard_normal((n, cols - 1)))
    w = rng.lognormal(0.0, 0.4, n) if weighted else None
    opt = pkg.make_options(tol=1e-8)
    a = absorber.absorb(y, X, fes, G, w, opt, save_fe=save)
    b = absorber.absorb(_pinned(y), _pinned(X), [_pinned(f) for f in fes], G, None if w is None else _pinned(w), opt,
                        y_out=_pinned(y), X_out=_pinned(X), save_fe=save)
    assert a.converged and b.converged and a.iterations == b.iterations
    assert np.array_equal(a.y_tilde, b.y_tilde) and np.array_equal(a.X_tilde, b.X_tilde)
    if save:
        assert all(np.array_equal(p, q) for p, q in zip(a.fe, b.fe))
    yi, Xi = y.copy(), X.copy(order="F")
    absorber.absorb(yi, Xi, fes, G, w, opt, y_out=yi, X_out=Xi, save_fe=save)
    assert np.array_equal(yi, a.y_tilde) and np.array_equal(Xi, a.X_tilde)


def test_threads_with_their_own_absorbers(pkg):
    """Two absorbers in two threads, both with staged copies, against one alone."""
    from concurrent.futures import ThreadPoolExecutor
    n, G = 400_000, [50_000, 4_000]
    rng = np.random.default_rng(0)
    fes = [rng.integers(0, g, n).astype(np.int32) for g in G]
    y, X = rng.standard_normal(n), np.asfortranarray(rng.standard_normal((n, 7)))
    opt = pkg.make_options(tol=1e-8)

    def run(_):
        a = pkg.Absorber(0)
        r = a.absorb(y, X, fes, G, None, opt)
        a.close()
        return r.y_tilde, r.X_tilde

    ref = run(0)
    with ThreadPoolExecutor(2) as ex:
        for out in ex.map(run, range(4)):
            assert np.array_equal(out[0], ref[0]) and np.array_equal(out[1], ref[1])
