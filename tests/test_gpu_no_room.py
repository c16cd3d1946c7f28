"""No room on the device for a faster form's workspace: the call takes the form that
needs less and gives the same answer.  B200FE_REFUSE at context creation refuses
the named workspace as a full device would.

Both forms stop at 1e-11 of ||b||; on these panels an error of the FE
coefficients shows up in the within transform less than a hundredfold, so 1e-9
of the column norm bounds the distance of either from the projection.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pair(pkg, monkeypatch, refuse, calls):
    """What each call gives with and without the refused workspace; the refusing context serves all calls."""
    monkeypatch.delenv("B200FE_REFUSE", raising=False)
    free = pkg.Absorber(0)
    monkeypatch.setenv("B200FE_REFUSE", refuse)
    tight = pkg.Absorber(0)
    monkeypatch.delenv("B200FE_REFUSE")
    out = [(c(free), c(tight)) for c in calls]
    free.close()
    tight.close()
    return out


def _same(a, b, y, X):
    assert a.converged and b.converged
    assert a.kernel_launches != b.kernel_launches  # another form
    for u, v, x in [(a.y_tilde, b.y_tilde, y[:, None])] + [(a.X_tilde, b.X_tilde, X)]:
        u, v = u.reshape(x.shape), v.reshape(x.shape)
        assert np.all(np.linalg.norm(u - v, axis=0) <= 1e-9 * np.linalg.norm(x, axis=0))


@pytest.mark.parametrize("refuse", ["pc_tile_val", "pc_key,pc32_,pc64_", "pc32_ctl,pc64_ctl"])
@pytest.mark.parametrize("years", [True, False])
def test_persistent_pcg(pkg, panels, monkeypatch, refuse, years):
    p = panels.akm_two_way(20_000, n_firms=600, n_years=12, seed=7, three_way=years)
    X = np.column_stack([p.X, np.random.default_rng(0).standard_normal((p.n, 4))])
    calls = [lambda a, k=k, c=c: a.absorb(p.y, X[:, :c], p.fes, p.levels, None, pkg.make_options(tol=1e-11, precision=k))
             for k in ("mixed", "fp64") for c in (2, 6)]
    for (a, b), c in zip(_pair(pkg, monkeypatch, refuse, calls), (2, 6, 2, 6)):
        _same(a, b, p.y, X[:, :c])


def test_tiles_of_both_precisions(pkg, panels):
    """The tiles of a reused structure are built for the second precision when it comes."""
    p = panels.akm_two_way(20_000, n_firms=600, n_years=12, seed=8, three_way=True)
    run = lambda a, k, reuse: a.absorb(p.y, p.X, p.fes, p.levels, None, pkg.make_options(  # noqa: E731
        tol=1e-9, precision=k, reuse_structure=reuse))
    both = pkg.Absorber(0)
    for i, k in enumerate(("mixed", "fp64", "mixed")):
        one = pkg.Absorber(0)
        a, b = run(one, k, False), run(both, k, i > 0)
        assert np.array_equal(a.y_tilde, b.y_tilde) and np.array_equal(a.X_tilde, b.X_tilde)
        one.close()
    both.close()


@pytest.mark.parametrize("refuse", ["sp_count", "sp_kin", "sp_val64", "run_meta1", "cfy32", "chunk_beg_sp"])
@pytest.mark.parametrize("years", [True, False])
def test_block_of_two_large_dims(pkg, panels, monkeypatch, refuse, years):
    if not years and refuse in ("run_meta1", "cfy32"):
        pytest.skip("no coupled small dim, no such workspace")
    p = panels.akm_two_way(20_000, n_firms=600, n_years=12, seed=9, three_way=True)
    rng = np.random.default_rng(9)
    spell = np.r_[True, (np.diff(p.fes[0]) != 0) | (np.diff(p.fes[1]) != 0)]
    job = rng.integers(0, 150, int(spell.sum()))[np.cumsum(spell) - 1].astype(np.int32)
    fes = [p.fes[0], p.fes[1], job] + ([p.fes[2]] if years else [])
    G = [int(f.max()) + 1 for f in fes]
    w = rng.lognormal(0.0, 0.5, p.n)
    calls = [lambda a, r=r: a.absorb(p.y, p.X, fes, G, w, pkg.make_options(tol=1e-11, precision="fp64",
                                                                       reuse_structure=r)) for r in (False, True)]
    (a, b), (_, again) = _pair(pkg, monkeypatch, refuse, calls)
    _same(a, b, p.y, p.X)
    assert again.setup_ms == 0.0 and np.array_equal(again.y_tilde, b.y_tilde)


def test_tile_records(pkg, panels, monkeypatch):
    p = panels.akm_two_way(60_000, n_firms=900, n_years=12, seed=10, three_way=True)
    call = lambda a: a.absorb(p.y, p.X, p.fes, p.levels, None, pkg.make_options(tol=1e-11))  # noqa: E731
    (a, b), = _pair(pkg, monkeypatch, "stream_blob", [call])
    _same(a, b, p.y, p.X)


@pytest.mark.parametrize("refuse", ["sl_xblk", "sl_xmom", "sl_xprim", "sl_xly", "sl_xpg", "sl_x"])
@pytest.mark.parametrize("cols", [1, 9])  # the form after a check interval, and at once
def test_slopes_in_coefficient_space(pkg, panels, monkeypatch, refuse, cols):
    p = panels.akm_two_way(30_000, n_firms=400, n_years=12, seed=11, three_way=True)
    rng = np.random.default_rng(11)
    z, X = rng.standard_normal(p.n), np.column_stack([p.X, rng.standard_normal((p.n, 6))])[:, : cols - 1]
    call = lambda a: a.absorb(p.y, X, p.fes, p.levels, None, pkg.make_options(tol=1e-11),  # noqa: E731
                              slopes=[(1, z, True)])
    (a, b), (_, again) = _pair(pkg, monkeypatch, refuse, [call, call])
    _same(a, b, p.y, X)
    assert np.array_equal(again.y_tilde, b.y_tilde) and again.kernel_launches == b.kernel_launches
