"""The interp bins that a 2-D plan chooses by taps, coils per block and sample density, on both
sides of each line of the rule, and that a plan changes them when its sample count does: against
the FP64 oracle, interp and coordinate gradients.

Tolerance: 2e-5 relative L2 (FP32 against the FP64 oracle), as for the other gridding kernels;
gradients against those of a plan whose caller chose the bins, 1e-5 (two FP32 sums of the same
terms in another order).
"""
import numpy as np
import pytest
import torch

import oracle as O
from mripy_gb300.plan import NufftPlan, Tuning

pytestmark = pytest.mark.gpu

EPS = {4: 1e-2, 6: 1e-3, 8: 1e-4, 10: 1e-5, 12: 5e-6, 14: 1e-6, 16: 5e-8, 28: 1e-15, 32: 1e-17}


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("W,nc,nt,dense,bins", [
    (4, 4, 12, False, (16, 16)), (4, 4, 12, True, (16, 16)), (4, 4, 3, False, (8, 16)), (6, 3, 12, False, (16, 16)),
    (8, 4, 12, False, (8, 16)), (12, 12, 5, False, (8, 16)), (14, 4, 12, True, (16, 16)), (16, 3, 12, False, (16, 16)),
    (10, 8, 12, False, (16, 16)), (10, 8, 12, True, (8, 16)), (10, 8, 4, False, (8, 16)), (12, 8, 12, False, (8, 16)),
    (16, 16, 5, False, (8, 16)), (12, 2, 9, True, (16, 16)), (12, 2, 8, True, (8, 16)), (6, 1, 12, False, (16, 16)),
    (28, 2, 2, False, (8, 16)), (32, 2, 2, False, (16, 16))])
def test_bins_and_interp(W, nc, nt, dense, bins):
    rng = np.random.default_rng(W + nc)
    shape = (40, 37)
    nsp, nf, tau = O.grid_params(2, *shape, eps=EPS[W])
    M = int(np.ceil((49 if dense else 10) * nf[0] * nf[1] / 128)) * nt
    p = NufftPlan(2, shape, n_coil=nc, n_traj=nt, eps=EPS[W])
    for m in (M, 300, M):  # the bins follow the samples; buffers are re-used
        off = [m * g // nt for g in range(nt + 1)]
        xs = rng.uniform(-np.pi, np.pi, (2, m))
        ks = [torch.from_numpy(v).cuda() for v in xs]
        p.set_points(ks, traj_offsets=off)
        if m == M:
            assert p.info()["nspread"] == nsp == W // 2 and p.info()["interp_tile"] == bins
        G = (rng.standard_normal((nt * nc,) + tuple(nf)) + 1j * rng.standard_normal((nt * nc,) + tuple(nf)))
        G = G.astype(np.complex64)
        g = torch.from_numpy(G).cuda()
        k = p.interp(g).cpu().numpy()
        for q in range(0, nt, max(1, nt // 2)):
            sl = slice(off[q], off[q + 1])
            ref = np.prod(nf) * O.interp(tuple(v[sl] for v in xs), G[q * nc:(q + 1) * nc], tau, nsp).T
            assert rel(k[sl], ref) < 2e-5
    if W <= 16:
        r = NufftPlan(2, shape, n_coil=nc, n_traj=nt, eps=EPS[W], tuning=Tuning(interp_tile=(12, 20)))
        r.set_points(ks, traj_offsets=off)
        c = torch.randn(M, nc, dtype=torch.complex64, device="cuda")
        a, b = p.interp_grad_coords(g, c).cpu().numpy(), r.interp_grad_coords(g, c).cpu().numpy()
        assert rel(a, b) < 1e-5
        r.close()
    p.close()
