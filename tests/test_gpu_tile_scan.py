"""set_points with more bins than one block scans (16,384): the chunked scan's lists, for bin
counts below, at and above one block's share, at the ends of chunks, and with chunks of several
steps (above 4,194,304 bins); the spread's tiles and the interp's bins are of different counts.

One cell per bin makes the bins many.  The type-2 transform of a group reads the interp's list,
the type-1 transform the spread's; an error in an offset moves samples between groups.

Tolerance: 2e-5 relative L2 (FP32 against the FP64 oracle), as for the other gridding tests.
"""
import numpy as np
import pytest
import torch

import oracle as O
from mripy_gb300.plan import NufftPlan, Tuning

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("groups,spread_tile,interp_tile", [
    (16, (32, 32), (1, 1)), (17, (1, 1), (32, 32)), (20, (1, 1), (1, 1)), (24, (2, 1), (1, 1)), (200, (1, 1), (4, 1)),
    (4100, (32, 32), (1, 1)), (4200, (1, 2), (1, 1))])
def test_lists_of_many_bins(groups, spread_tile, interp_tile):
    rng = np.random.default_rng(groups)
    shape, counts = (16, 16), rng.integers(0, 6, groups)
    counts[[0, groups // 2, groups - 1]] = 0, 700, 5
    off = np.concatenate([[0], np.cumsum(counts)])
    M = int(off[-1])
    xs = rng.uniform(-np.pi, np.pi, (2, M))
    p = NufftPlan(2, shape, n_traj=groups, eps=1e-3,
                  tuning=Tuning(spread_tile=spread_tile, interp_tile=interp_tile, max_subproblem=16))
    p.set_points([torch.from_numpy(v).cuda() for v in xs], traj_offsets=off.tolist())
    assert p.info()["nf"] == (32, 32)
    c = (rng.standard_normal((M, 1)) + 1j * rng.standard_normal((M, 1))).astype(np.complex64)
    F = p.type1(torch.from_numpy(c).cuda()).cpu().numpy()
    k = p.type2(torch.from_numpy(F).cuda()).cpu().numpy()
    assert np.all(F[counts == 0] == 0) and np.isfinite(F.view(np.float32)).all()
    for g in np.unique(np.concatenate([np.flatnonzero(counts)[:: max(1, groups // 40)], [groups // 2, groups - 1]])):
        sl = slice(off[g], off[g + 1])
        xg = tuple(v[sl] for v in xs)
        Fo = O.nufft_type1(xg, c[sl].astype(np.complex128), shape, eps=1e-3)
        ko = O.nufft_type2(xg, F[g].astype(np.complex128), shape, eps=1e-3)
        assert np.linalg.norm(F[g] - Fo) < 2e-5 * np.linalg.norm(Fo)
        assert np.linalg.norm(k[sl] - ko) < 2e-5 * np.linalg.norm(ko)
    p.close()
