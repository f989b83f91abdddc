"""set_points: the cell of every sample as Python's % and // choose it, and the work lists.

Cells: one group per sample, so that each spread grid shows one stencil; its non-zero cells have
to be exactly the oracle's (a cell one off would move the stencil's edge).  Coordinates at, one
ulp below and one above whole cells and whole turns, zeros of both signs, far outside
(-2 pi, 2 pi), in both types and with df = 2.

Lists: the totals that set_points reads back and the transforms on them, for tile counts below,
at and above one step of the scan (4096 tiles), with empty groups, dense tiles and a re-used
plan whose sample count shrinks and grows.
"""
import numpy as np
import pytest
import torch

import oracle as O
from mripy_gb300 import _native as N
from mripy_gb300.plan import NufftPlan, Tuning

pytestmark = pytest.mark.gpu


def _coordinates(nf, rng):
    h = 2 * np.pi / nf
    v = [0.0, -0.0, np.pi, -np.pi, 2 * np.pi, -2 * np.pi, 6.5, -6.5, 1e3, -1e3, 1e-300, -1e-300, 1e-17, -1e-17]
    for k in list(range(0, nf, 3)) + [nf - 1, nf, nf + 1]:
        for s in (1, -1):
            for x in (s * k * h, s * k * h - 2 * np.pi):
                v += [x, np.nextafter(x, 10), np.nextafter(x, -10)]
    return np.concatenate([v, rng.uniform(-8, 8, 200)])


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("ms,df", [(16, 1.0), (27, 1.0), (50, 2.0)])
def test_cells_of_every_sample(dtype, ms, df):
    rng = np.random.default_rng(ms)
    nsp, nf, tau = O.grid_params(1, ms, eps=5e-6)
    x = _coordinates(nf[0], rng).astype(dtype)
    K = len(x)
    p = NufftPlan(1, (ms,), n_traj=K, eps=5e-6, df=df).set_points([torch.from_numpy(x).cuda()],
                                                                  traj_offsets=list(range(K + 1)))
    g = p.spread(torch.ones(K, 1, dtype=torch.complex64, device="cuda")).cpu().numpy()
    for k in range(K):
        ref = O.spread((x[k:k + 1].astype(np.float64) * df,), np.ones((1, 1), np.complex128), tau, nsp, nf)[0]
        assert np.array_equal(g[k] != 0, ref != 0), (k, x[k])
        assert np.abs(g[k] - ref).max() < 2e-6
    p.close()


def test_wide_axis_cells():
    """More cells than an FP32 estimate places within one (1-D)."""
    ms = 1 << 20
    nsp, nf, tau = O.grid_params(1, ms, eps=1e-3)
    rng = np.random.default_rng(1)
    h = 2 * np.pi / nf[0]
    k = rng.integers(0, nf[0], 200)
    x = np.concatenate([k * h, np.nextafter(k * h, 0), rng.uniform(-np.pi, np.pi, 200)])
    p = NufftPlan(1, (ms,), eps=1e-3).set_points([torch.from_numpy(x).cuda()])
    c = (rng.standard_normal((len(x), 1)) + 1j).astype(np.complex64)
    g = p.spread(torch.from_numpy(c).cuda()).cpu().numpy()
    ref = O.spread((x,), c.T.astype(np.complex128), tau, nsp, nf)
    assert np.linalg.norm(g - ref) < 2e-5 * np.linalg.norm(ref)
    p.close()


@pytest.mark.parametrize("groups,shape", [(1, (32, 32)), (16, (128, 128)), (17, (128, 128)), (40, (96, 80))])
def test_lists_and_transforms(groups, shape):
    rng = np.random.default_rng(groups)
    counts = rng.integers(0, 400, groups)
    counts[groups // 2] = 0 if groups > 1 else 300
    p = NufftPlan(2, shape, n_traj=groups, eps=5e-6, tuning=Tuning(max_subproblem=64))
    for scale in (1.0, 0.3, 2.0):  # the plan's buffers are re-used
        off = np.concatenate([[0], np.cumsum((counts * scale).astype(int))])
        M = int(off[-1])
        xs = rng.uniform(-np.pi, np.pi, (2, M))
        xs[:, ::3] *= 0.02
        p.set_points([torch.from_numpy(v).cuda() for v in xs], traj_offsets=off.tolist())
        inf = p.info()
        assert inf["n_samples"] == M and inf["spread_entries"] >= M
        c = (rng.standard_normal((M, 1)) + 1j * rng.standard_normal((M, 1))).astype(np.complex64)
        F = p.type1(torch.from_numpy(c).cuda()).cpu().numpy()
        k = p.type2(torch.from_numpy(F).cuda()).cpu().numpy()
        for g in range(0, groups, max(1, groups // 4)):
            sl = slice(off[g], off[g + 1])
            if off[g] == off[g + 1]:
                assert np.all(F[g] == 0)
                continue
            xg = tuple(v[sl] for v in xs)
            Fo = O.nufft_type1(xg, c[sl].astype(np.complex128), shape, eps=5e-6)
            ko = O.nufft_type2(xg, F[g].astype(np.complex128), shape, eps=5e-6)
            assert np.linalg.norm(F[g] - Fo) < 2e-5 * np.linalg.norm(Fo)
            assert np.linalg.norm(k[sl] - ko) < 2e-5 * np.linalg.norm(ko)
    p.close()


def test_non_finite_coordinates_refused_and_plan_usable_after():
    p = NufftPlan(2, (32, 32), eps=5e-6)
    x = torch.rand(100, dtype=torch.float64, device="cuda")
    for bad in (float("nan"), float("inf"), -float("inf")):
        y = x.clone()
        y[57] = bad
        with pytest.raises(N.GbnError):
            p.set_points([x, y])
        with pytest.raises(N.GbnError):
            N.check(N.lib().gbn_type1(p._h, x.data_ptr(), N.Layout(0, 1, 1), None, x.data_ptr(), N.Layout(0, 1, 1), None))
    p.set_points([x, x])
    c = torch.ones(100, 1, dtype=torch.complex64, device="cuda")
    assert torch.isfinite(torch.view_as_real(p.type1(c))).all()
    p.close()
