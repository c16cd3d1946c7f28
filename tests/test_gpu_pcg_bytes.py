"""Algorithmic bytes that the profile gives for the persistent PCG: per iteration the block's
nonzeros (column id and value), its row offsets, p gathered and q written once, the
coupling rows, and the vectors as the two updates read and write them: r, q -> r and
r, p, x -> x, p, with the diagonal in each."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,size", [("mixed", 4), ("fp64", 8)])
@pytest.mark.parametrize("cols,pitch", [(3, 4), (7, 8), (13, 16)])
@pytest.mark.parametrize("years", [0, 10])
def test_bytes_of_an_iteration(absorber, pkg, precision, size, cols, pitch, years):
    rng = np.random.default_rng(cols)
    firms, workers = 100, 1_500
    pair = np.stack([rng.integers(0, firms - 1, workers), rng.integers(0, firms - 1, workers)])
    pair[1] += pair[1] >= pair[0]  # two distinct firms each
    worker = np.repeat(np.arange(workers), 6).astype(np.int32)
    firm = np.repeat(pair.T, 3, axis=1).ravel().astype(np.int32)
    fes, G = [worker, firm], [workers, firms]
    if years:
        fes, G = fes + [rng.integers(0, years, worker.size).astype(np.int32)], G + [years]
    assert np.unique(firm).size == firms
    import torch
    v = torch.from_numpy(rng.standard_normal((cols, worker.size))).cuda()
    _, r = absorber.absorb_device(v, [torch.from_numpy(f).cuda() for f in fes], G, None,
                                  pkg.make_options(tol=1e-9, precision=precision, profile=True))
    assert r.converged and r.iterations > 0
    nnz = firms + 2 * np.unique(np.sort(pair, axis=0), axis=1).shape[1]
    rows = firms + years
    want = nnz * (4 + size) + firms * 4 + 2 * firms * pitch * size + firms * ((years + 3) // 4 * 4) * size \
        + 8 * rows * pitch * size + 2 * rows * size
    assert r.prof_bytes[0] == pytest.approx(r.iterations * want, rel=1e-12)
