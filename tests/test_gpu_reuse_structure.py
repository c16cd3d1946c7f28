"""reuse_structure with two large dims beside the primary: the structure differs by
precision, and a call that reuses one gives the same bits as the same call of a
fresh context, whichever precision the calls before it had; a call like the one
before it builds nothing."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _panel(panels, years):
    p = panels.akm_two_way(20_000, n_firms=500, n_years=12, seed=4, three_way=True)
    rng = np.random.default_rng(4)
    job = rng.integers(0, 90, 40_000)[(p.fes[0].astype(np.int64) * 3 + p.fes[1]) % 40_000]
    fes = [p.fes[0], p.fes[1], job.astype(np.int32)] + ([p.fes[2]] if years else [])
    return p, fes, [int(f.max()) + 1 for f in fes]


@pytest.mark.parametrize("years", [True, False])
@pytest.mark.parametrize("order", ["mffm", "fmmf", "mfmf"])
def test_answers_do_not_depend_on_earlier_calls(pkg, panels, order, years):
    p, fes, G = _panel(panels, years)
    opt = {k: dict(tol=1e-9, precision=v) for k, v in {"m": "mixed", "f": "fp64"}.items()}
    alone = {}
    for k in "mf":
        a = pkg.Absorber(0)
        alone[k] = a.absorb(p.y, p.X, fes, G, None, pkg.make_options(**opt[k]))
        a.close()
    a = pkg.Absorber(0)
    for i, k in enumerate(order):
        r = a.absorb(p.y, p.X, fes, G, None, pkg.make_options(**opt[k], reuse_structure=True))
        assert r.converged and r.iterations == alone[k].iterations
        assert np.array_equal(r.y_tilde, alone[k].y_tilde) and np.array_equal(r.X_tilde, alone[k].X_tilde)
        assert (r.setup_ms == 0.0) == (i > 0 and order[i - 1] == k)
    a.close()


def test_device_calls_and_one_large_dim(pkg, panels):
    import torch
    p, fes, G = _panel(panels, True)
    v = torch.from_numpy(np.column_stack([p.y, p.X]).T.copy()).cuda()
    for dims in ((0, 1, 2, 3), (0, 1, 3)):
        ids, lv = [torch.from_numpy(fes[d]).cuda() for d in dims], [G[d] for d in dims]
        alone, a = {}, pkg.Absorber(0)
        for k in ("mixed", "fp64"):
            b = pkg.Absorber(0)
            alone[k] = b.absorb_device(v, ids, lv, None, pkg.make_options(tol=1e-9, precision=k))[0].cpu()
            b.close()
        for i, k in enumerate(("fp64", "mixed", "mixed", "fp64")):
            out, r = a.absorb_device(v, ids, lv, None, pkg.make_options(tol=1e-9, precision=k, reuse_structure=True))
            assert torch.equal(out.cpu(), alone[k])
            if len(dims) == 3:  # one large dim: one structure for both
                assert (r.setup_ms == 0.0) == (i > 0)
        a.close()
