"""The 3-D kernels for 1 to 3 coils -- the register-tile spread (k_spread3d_few) and the
one-coil-per-block interp with paired cells (k_interp3d_one) -- against the FP64 oracle.

Covered: every coil count they take, stencils of 6 to 14 taps (the lane layouts of 10 taps, of
other multiples of 4 and of the rest), odd oversampled grids (partial edge tiles, unpaired grid
reads), stencils across the periodic edge, split tiles, bins above and below the staging
threshold, several trajectory groups with an empty one, density weights, strided samples, a
grid buffer off a 16-byte boundary, real-valued samples (density compensation) and samples or
grid cells that are not finite.

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
    xs = rng.uniform(-np.pi, np.pi, (3, M))
    xs[:, :M // 3] *= 0.08                                  # dense centre: split tiles, long bins
    xs[:, M // 3:M // 3 + 50] = np.pi                       # stencils across the periodic edge
    return xs


@pytest.mark.parametrize("nc", [1, 2, 3])
@pytest.mark.parametrize("eps,ns", [(1e-3, 3), (1e-4, 4), (1e-5, 5), (5e-6, 6), (1e-6, 7), (1e-7, 8)])
def test_few_coils_gridding_against_oracle(nc, eps, ns):
    rng = np.random.default_rng(100 * ns + nc)
    M, shape = 5001, (26, 25, 23)
    xs = _points(rng, M)
    p = NufftPlan(3, shape, n_coil=nc, eps=eps).set_points([cuda(v) for v in xs])
    assert p.info()["nspread"] == ns and p.info()["spread_tile"] == (8, 8, 16 if nc == 1 else 8)
    nsp, nf, tau = O.grid_params(3, *shape, eps=eps)
    c = cvec(rng, (M, nc))
    g = p.spread(cuda(c)).clone()
    assert rel(g, O.spread(tuple(xs), c.T, tau, nsp, nf)) < TOL_REF
    G = cvec(rng, (nc,) + nf)
    out = p.interp(cuda(G))
    assert rel(out, np.prod(nf) * O.interp(tuple(xs), G, tau, nsp).T) < TOL_REF
    assert torch.equal(out, p.interp(cuda(G)))              # summed in a fixed order
    p.close()


@pytest.mark.parametrize("nc", [1, 2, 3])
@pytest.mark.parametrize("shape,eps", [((21, 19, 17), 1e-12), ((64, 64, 64), 5e-6)])
def test_few_coils_transforms_groups_and_strides(nc, shape, eps):
    """Odd grids (ratio 3) and sparse bins; three groups, one empty; weights; coil-major
    samples; transforms equal the oracle's per group."""
    rng = np.random.default_rng(nc)
    off = [0, 1300, 1300, 4000]
    M = off[-1]
    xs = _points(rng, M)
    w = rng.uniform(0.5, 1.5, M).astype(np.float32)
    p = NufftPlan(3, shape, n_coil=nc, n_traj=3, eps=eps, max_nspread=6)
    p.set_points([cuda(v) for v in xs], traj_offsets=off)
    c, img = cvec(rng, (M, nc)), cvec(rng, (3,) + shape + (nc,))
    cm = cuda(np.ascontiguousarray(c.T)).t()                # coil stride M
    F = p.type1(cm, weight=cuda(w)).cpu().numpy()
    km = torch.empty((nc, M), dtype=torch.complex64, device="cuda").t()
    k = p.type2(cuda(img), out=km).cpu().numpy()
    n21 = p.type21(cuda(img), dcf=cuda(w)).cpu().numpy()
    for g in (0, 2):
        sl = slice(off[g], off[g + 1])
        xg = tuple(v[sl] for v in xs)
        cw = (c[sl] * w[sl, None]).astype(np.complex128)
        assert rel(F[g], O.nufft_type1(xg, cw, shape, eps=eps)) < TOL_REF
        ko = O.nufft_type2(xg, img[g].astype(np.complex128), shape, eps=eps)
        assert rel(k[sl], ko) < TOL_REF
        assert rel(n21[g], O.nufft_type1(xg, ko * w[sl, None], shape, eps=eps)) < TOL_REF
    assert np.all(F[1] == 0)
    p.close()


def test_few_coils_unaligned_grid_long_items_and_explicit_tiles():
    """A grid 8 bytes past a 16-byte boundary (unpaired reads), items of 64 and 4096 samples,
    and the kernels a caller's own tiles select agree with the defaults."""
    rng = np.random.default_rng(5)
    M, shape = 9000, (24, 24, 24)
    xs = _points(rng, M)
    c = cuda(cvec(rng, (M, 1)))
    ref = NufftPlan(3, shape, eps=5e-6).set_points([cuda(v) for v in xs])
    g0 = ref.spread(c).clone()
    k0 = ref.interp(g0)
    buf = torch.empty(g0.numel() + 1, dtype=torch.complex64, device="cuda")
    view = buf[1:].view(g0.shape)
    assert view.data_ptr() % 16 == 8
    view.copy_(g0)
    assert float((ref.interp(view) - k0).abs().max()) <= 1e-6 * float(k0.abs().max())
    for tu in (Tuning(max_subproblem=64), Tuning(max_subproblem=4096), Tuning(spread_tile=(8, 8, 32)),
               Tuning(interp_tile=(16, 16, 24))):
        p = NufftPlan(3, shape, eps=5e-6, tuning=tu).set_points([cuda(v) for v in xs])
        assert float((p.spread(c) - g0).abs().max()) <= 2e-5 * float(g0.abs().max())
        assert float((p.interp(g0) - k0).abs().max()) <= 2e-5 * float(k0.abs().max())
        p.close()


@pytest.mark.parametrize("nc", [1, 3])
def test_few_coils_non_finite_values_stay_in_their_stencil(nc):
    rng = np.random.default_rng(9)
    M, shape = 3000, (24, 24, 24)
    xs = rng.uniform(-np.pi, np.pi, (3, M))
    p = NufftPlan(3, shape, n_coil=nc, eps=5e-6).set_points([cuda(v) for v in xs])
    c = cvec(rng, (M, nc))
    g0 = p.spread(cuda(c)).cpu().numpy().copy()
    ones = np.zeros((M, nc), np.complex64)
    ones[77] = 1.0
    inside = np.abs(p.spread(cuda(ones)).cpu().numpy()) > 0
    assert inside.sum() == nc * 12 ** 3
    c[77] = np.inf
    g1 = p.spread(cuda(c)).cpu().numpy()
    assert np.array_equal(np.isfinite(g1), ~inside)
    assert np.array_equal(g1[~inside], g0[~inside]) or rel(g1[~inside], g0[~inside]) < 1e-6
    G = cvec(rng, g0.shape)
    k0 = p.interp(cuda(G)).cpu().numpy()
    cell = tuple(np.argwhere(inside[0])[0])
    G[(slice(None),) + cell] = np.nan
    k1 = p.interp(cuda(G)).cpu().numpy()
    assert not np.isfinite(k1[77]).any()
    touched = ~np.isfinite(k1)
    assert 1 <= touched[:, 0].sum() < 200
    assert np.array_equal(k1[~touched], k0[~touched])
    p.close()


def test_few_coils_real_samples_match_complex():
    """The density compensation's real-valued spread gives the complex spread's iterates."""
    rng = np.random.default_rng(11)
    M, shape = 6000, (24, 22, 20)
    xs = _points(rng, M)
    p = NufftPlan(3, shape, eps=5e-6).set_points([cuda(v) for v in xs])
    d = p.pipe_menon_dcf(3).cpu().numpy()
    w = torch.ones((M, 1), dtype=torch.complex64, device="cuda")
    for _ in range(3):
        w = w / p.interp(p.spread(w)).abs()
    w = w.real.cpu().numpy()[:, 0]
    assert rel(d, w * M / w.sum()) < TOL_REF
    p.close()


@pytest.mark.parametrize("eps,ns", [(1e-3, 3), (1e-4, 4), (1e-5, 5), (5e-6, 6), (1e-6, 7)])
def test_one_coil_interp_samples_in_every_cell_of_a_bin(eps, ns):
    """Staged bins with samples in their last cells, where the lane past the last tap would read
    behind the window (even tiles whose window starts on an odd cell)."""
    rng = np.random.default_rng(ns)
    M, shape = 30000, (16, 16, 16)
    xs = rng.uniform(-np.pi, np.pi, (3, M))
    p = NufftPlan(3, shape, eps=eps).set_points([cuda(v) for v in xs])
    nsp, nf, tau = O.grid_params(3, *shape, eps=eps)
    assert nsp == ns and M > 64 * p.info()["interp_subproblems"]
    G = cvec(rng, (1,) + nf)
    assert rel(p.interp(cuda(G)), np.prod(nf) * O.interp(tuple(xs), G, tau, nsp).T) < TOL_REF
    p.close()


@pytest.mark.parametrize("nc", [4, 5, 6])
@pytest.mark.parametrize("shape,eps", [((26, 25, 24), 1e-5), ((19, 18, 17), 1e-12), ((24, 24, 24), 5e-6), ((22, 20, 24), 1e-3)])
def test_four_to_six_coils_interp_against_oracle(nc, shape, eps):
    """These run one coil per block too: staged and sparse bins, two groups, odd grids, coil-major
    samples, and the caller's own coil group agrees."""
    rng = np.random.default_rng(nc)
    off = [0, 3000, 9000]
    M = off[-1]
    xs = _points(rng, M)
    p = NufftPlan(3, shape, n_coil=nc, n_traj=2, eps=eps, max_nspread=6)
    p.set_points([cuda(v) for v in xs], traj_offsets=off)
    nsp, nf, tau = O.grid_params(3, *shape, eps=eps, max_nspread=6)
    assert p.info()["interp_coil_group"] == 1
    G = cvec(rng, (2, nc) + nf)
    km = torch.empty((nc, M), dtype=torch.complex64, device="cuda").t()
    k = p.interp(cuda(G), out=km).cpu().numpy()
    for g in (0, 1):
        sl = slice(off[g], off[g + 1])
        ref = np.prod(nf) * O.interp(tuple(v[sl] for v in xs), G[g], tau, nsp).T
        assert rel(k[sl], ref) < TOL_REF
    q = NufftPlan(3, shape, n_coil=nc, n_traj=2, eps=eps, max_nspread=6, tuning=Tuning(interp_coil_group=4))
    q.set_points([cuda(v) for v in xs], traj_offsets=off)
    assert rel(q.interp(cuda(G)), k) < 2e-6
    p.close()
    q.close()
