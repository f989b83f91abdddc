"""The density compensation's interp of a real grid (k_interp3d_real) against the complex interp.

Tolerance: 2e-5 relative L2, as for the other gridding kernels.
"""
import numpy as np
import pytest
import torch

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


@pytest.mark.parametrize("eps,ns", [(1e-3, 3), (1e-4, 4), (1e-5, 5), (5e-6, 6)])
@pytest.mark.parametrize("tile", [(8, 8, 8), (5, 6, 11), (4, 9, 16)])
def test_density_real_grid_interp_matches_complex(eps, ns, tile):
    """The density compensation's interp of a real grid (the lane tables of 6 to 12 taps, tiles
    of other sizes, bins that start on odd cells, two groups) against the complex interp."""
    rng = np.random.default_rng(10 * ns + tile[0])
    off = [0, 14000, 30000]
    M, shape = off[-1], (24, 22, 20)
    xs = _points(rng, M)
    p = NufftPlan(3, shape, n_traj=2, eps=eps, tuning=Tuning(interp_tile=tile))
    p.set_points([cuda(v) for v in xs], traj_offsets=off)
    inf = p.info()
    assert inf["nspread"] == ns and inf["nf"][2] % 2 == 0 and M >= 24 * inf["interp_subproblems"]
    d = p.pipe_menon_dcf(2).cpu().numpy()
    w = torch.ones((M, 1), dtype=torch.complex64, device="cuda")
    for _ in range(2):
        w = w / p.interp(p.spread(w)).abs()
    w = w.real.cpu().numpy()[:, 0]
    for g in (0, 1):
        sl = slice(off[g], off[g + 1])
        assert rel(d[sl], w[sl] * (off[g + 1] - off[g]) / w[sl].sum()) < TOL_REF
    p.close()
