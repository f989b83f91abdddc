"""3-D interps of 2 to 5 coils on both sides of the lines between a block per coil and groups of
coils that depend on the coils' own grid size: against the FP64 oracle.

Tolerance: 2e-5 relative L2 (FP32 against the FP64 oracle), as for the other gridding kernels.
"""
import numpy as np
import pytest
import torch

import oracle as O
from mripy_gb300.plan import NufftPlan

pytestmark = pytest.mark.gpu

EPS = {6: 1e-3, 8: 1e-4, 12: 5e-6, 14: 1e-6}


@pytest.mark.parametrize("W,nc,n,M,nt,cg", [
    (6, 2, 32, 65536, 1, 1), (6, 2, 32, 65537, 1, 2), (6, 3, 32, 40000, 23, 1), (6, 3, 32, 60000, 24, 4),
    (6, 3, 32, 12000, 24, 1), (6, 3, 32, 393216, 24, 1), (6, 5, 32, 60000, 8, 1), (6, 5, 32, 60000, 9, 8),
    (8, 3, 32, 30000, 16, 1), (8, 3, 32, 30000, 17, 4), (8, 3, 32, 2200, 17, 1), (8, 3, 32, 278528, 17, 1),
    (8, 4, 32, 92160, 9, 1), (8, 4, 32, 92159, 9, 4), (8, 4, 32, 200000, 16, 4),
    (12, 3, 32, 30000, 32, 1), (12, 3, 32, 30000, 33, 4), (12, 3, 32, 4000, 33, 1), (12, 3, 32, 270336, 33, 1),
    (12, 4, 32, 100000, 16, 4), (12, 4, 32, 196608, 16, 1),
    (14, 3, 32, 30000, 8, 4), (14, 3, 32, 3800, 8, 1), (14, 3, 32, 131072, 8, 1), (14, 3, 32, 2200, 16, 1),
    (14, 3, 32, 20000, 16, 4)])
def test_interp_groups_by_grid_size(W, nc, n, M, nt, cg):
    rng = np.random.default_rng(W * nc + nt)
    shape = (n,) * 3
    nsp, nf, tau = O.grid_params(3, *shape, eps=EPS[W])
    off = [M * g // nt for g in range(nt + 1)]
    xs = rng.uniform(-np.pi, np.pi, (3, M))
    p = NufftPlan(3, shape, n_coil=nc, n_traj=nt, eps=EPS[W])
    p.set_points([torch.from_numpy(v).cuda() for v in xs], traj_offsets=off)
    assert 2 * nsp == W and p.info()["interp_coil_group"] == cg
    gen = torch.Generator(device="cuda").manual_seed(1)
    g = torch.randn((nt * nc,) + tuple(nf), generator=gen, dtype=torch.complex64, device="cuda")
    k = p.interp(g).cpu().numpy()
    for q in (0, nt - 1):
        take = np.arange(off[q], off[q + 1])[:: max(1, (off[q + 1] - off[q]) // 500)]
        ref = np.prod(nf) * O.interp(tuple(v[take] for v in xs), g[q * nc:(q + 1) * nc].cpu().numpy(), tau, nsp).T
        assert np.linalg.norm(k[take] - ref) < 2e-5 * np.linalg.norm(ref)
    p.close()
