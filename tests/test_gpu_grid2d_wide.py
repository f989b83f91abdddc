"""2-D gridding with wide stencils (k_spread2d_wide, k_interp2d_wide: 18 to 30 taps per axis, the
functions' default accuracy among them) against the FP64 oracle.

Covered: the narrowest, the default and the widest stencils they take and the next ones on either
side (other kernels), odd grids (unpaired reads, partial edge tiles), stencils across the
periodic edge, split tiles, several coils and groups with an empty one, weights, a grid off a
16-byte boundary, the smallest grid they take and one below, values that are not finite.

Tolerance: 2e-5 relative L2 (FP32 against the FP64 oracle), as for the other gridding kernels.
"""
import numpy as np
import pytest
import torch

import oracle as O
from mripy_gb300.plan import NufftPlan, Tuning

pytestmark = pytest.mark.gpu

TOL_REF = 2e-5


def cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda")


def cvec(rng, shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)


def rel(a, b):
    a = a.cpu().numpy() if isinstance(a, torch.Tensor) else np.asarray(a)
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def _points(rng, M):
    xs = rng.uniform(-np.pi, np.pi, (2, M))
    xs[:, :M // 3] *= 0.05
    xs[:, M // 3:M // 3 + 40] = np.pi
    return xs


# eps -> nspread 8 (narrower kernel), 9, 10, 14 (default), 15, 16 (wider: the general kernel)
@pytest.mark.parametrize("eps,ns", [(5e-8, 8), (6e-9, 9), (1e-11 * 1.5, 12), (2e-13, 12), (1e-15, 14), (1e-16, 15), (1e-17, 16)])
@pytest.mark.parametrize("shape", [(40, 40), (37, 33), (20, 20), (22, 21)])
def test_wide_gridding_against_oracle(eps, ns, shape):
    rng = np.random.default_rng(ns)
    M = 2500
    xs = _points(rng, M)
    p = NufftPlan(2, shape, n_coil=2, eps=eps).set_points([cuda(v) for v in xs])
    nsp, nf, tau = O.grid_params(2, *shape, eps=eps)
    assert p.info()["nspread"] == nsp == ns
    if 9 <= ns <= 15:
        assert (p.info()["spread_tile"] == (32, 32)) == (min(nf) >= 32 + 2 * ns)
    c = cvec(rng, (M, 2))
    assert rel(p.spread(cuda(c)), O.spread(tuple(xs), c.T, tau, nsp, nf)) < TOL_REF
    G = cvec(rng, (2,) + nf)
    assert rel(p.interp(cuda(G)), np.prod(nf) * O.interp(tuple(xs), G, tau, nsp).T) < TOL_REF
    p.close()


@pytest.mark.parametrize("nc", [1, 3])
def test_wide_groups_weights_and_layouts(nc):
    rng = np.random.default_rng(nc)
    shape, off = (32, 30), [0, 900, 900, 2300]
    M = off[-1]
    xs = _points(rng, M)
    w = rng.uniform(0.5, 1.5, M).astype(np.float32)
    p = NufftPlan(2, shape, n_coil=nc, n_traj=3, tuning=Tuning(max_subproblem=100)).set_points(
        [cuda(v) for v in xs], traj_offsets=off)
    c, img = cvec(rng, (M, nc)), cvec(rng, (3,) + shape + (nc,))
    F = p.type1(cuda(np.ascontiguousarray(c.T)).t(), weight=cuda(w)).cpu().numpy()
    k = p.type2(cuda(img)).cpu().numpy()
    n21 = p.type21(cuda(img), dcf=cuda(w)).cpu().numpy()
    for g in (0, 2):
        sl = slice(off[g], off[g + 1])
        xg = tuple(v[sl] for v in xs)
        assert rel(F[g], O.nufft_type1(xg, (c[sl] * w[sl, None]).astype(np.complex128), shape, eps=1e-15)) < TOL_REF
        ko = O.nufft_type2(xg, img[g].astype(np.complex128), shape, eps=1e-15)
        assert rel(k[sl], ko) < TOL_REF
        assert rel(n21[g], O.nufft_type1(xg, ko * w[sl, None], shape, eps=1e-15)) < TOL_REF
    assert np.all(F[1] == 0)
    p.close()


def test_wide_unaligned_grid_and_non_finite():
    rng = np.random.default_rng(3)
    M, shape = 1500, (40, 40)
    xs = rng.uniform(-np.pi, np.pi, (2, M))
    p = NufftPlan(2, shape).set_points([cuda(v) for v in xs])
    c = cvec(rng, (M, 1))
    g0 = p.spread(cuda(c)).clone()
    k0 = p.interp(g0).cpu().numpy()
    buf = torch.empty(g0.numel() + 1, dtype=torch.complex64, device="cuda")
    view = buf[1:].view(g0.shape)
    view.copy_(g0)
    assert rel(p.interp(view), k0) < 1e-6
    one = np.zeros((M, 1), np.complex64)
    one[7] = 1.0
    inside = p.spread(cuda(one)).cpu().numpy() != 0
    assert inside.sum() == 28 * 28
    c[7] = np.nan
    g1 = p.spread(cuda(c)).cpu().numpy()
    assert np.array_equal(np.isfinite(g1), ~inside)
    g = g0.cpu().numpy()
    g[(0,) + tuple(np.argwhere(inside[0])[0])] = np.inf
    k1 = p.interp(cuda(g)).cpu().numpy()
    touched = ~np.isfinite(k1)
    assert touched[7, 0] and touched.sum() < 400
    assert np.array_equal(k1[~touched], k0[~touched])
    p.close()


@pytest.mark.parametrize("eps,ns", [(6e-9, 9), (2e-13, 12), (1e-15, 14), (1e-16, 15)])
def test_wide_interp_samples_in_every_cell_of_a_bin(eps, ns):
    """Samples in the bins' last cells, where the lane past the last tap would read behind the
    window (even tiles whose window starts on an odd cell)."""
    rng = np.random.default_rng(ns)
    M, shape = 20000, (20, 20)
    xs = rng.uniform(-np.pi, np.pi, (2, M))
    p = NufftPlan(2, shape, eps=eps).set_points([cuda(v) for v in xs])
    nsp, nf, tau = O.grid_params(2, *shape, eps=eps)
    assert nsp == ns
    G = cvec(rng, (1,) + nf)
    assert rel(p.interp(cuda(G)), np.prod(nf) * O.interp(tuple(xs), G, tau, nsp).T) < TOL_REF
    p.close()
