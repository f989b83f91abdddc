"""3-D interps of 1 to 7 coils on both sides of the lines between a block per coil and groups of
coils (the taps, the coils, the samples and bins of the plan decide), and coordinate gradients on
both sides of theirs, against the FP64 oracle and a plan whose caller chose the group.

Tolerance: 2e-5 relative L2 (FP32 against the FP64 oracle), as for the other gridding kernels;
gradients against another group size, 1e-5 (two FP32 sums of the same terms in another order).
"""
import numpy as np
import pytest
import torch

import oracle as O
from mripy_gb300.plan import NufftPlan, Tuning

pytestmark = pytest.mark.gpu

EPS = {4: 1e-2, 6: 1e-3, 8: 1e-4, 10: 1e-5, 12: 5e-6, 14: 1e-6}


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("W,nc,n,M,nt,cg", [
    (4, 6, 16, 5461, 1, 1), (4, 6, 16, 5462, 1, 8), (4, 2, 20, 17000, 1, 2), (4, 1, 16, 40000, 1, 1),
    (4, 2, 72, 40000, 1, 1), (6, 4, 16, 65536, 1, 1), (6, 4, 16, 65600, 1, 4), (6, 1, 16, 300000, 1, 1),
    (8, 4, 32, 9000, 8, 1), (8, 4, 32, 9000, 9, 4), (8, 3, 32, 9000, 9, 1), (10, 6, 32, 9216, 9, 1),
    (8, 4, 32, 1500, 9, 1), (12, 5, 32, 36000, 9, 1), (12, 4, 32, 2000, 9, 1),
    (14, 4, 32, 1000, 8, 1), (12, 4, 32, 36900, 9, 1), (12, 4, 32, 36000, 9, 4), (14, 5, 32, 4000, 7, 1),
    (14, 5, 32, 4000, 8, 8), (14, 6, 16, 262200, 64, 1), (14, 4, 32, 4000, 8, 4), (14, 3, 32, 4000, 8, 1),
    (12, 7, 16, 3000, 1, 8)])
def test_interp_groups(W, nc, n, M, nt, cg):
    rng = np.random.default_rng(W * nc)
    shape = (n,) * 3
    nsp, nf, tau = O.grid_params(3, *shape, eps=EPS[W])
    off = [M * g // nt for g in range(nt + 1)]
    xs = rng.uniform(-np.pi, np.pi, (3, M))
    xs[:, ::5] *= 0.05
    p = NufftPlan(3, shape, n_coil=nc, n_traj=nt, eps=EPS[W])
    p.set_points([torch.from_numpy(v).cuda() for v in xs], traj_offsets=off)
    assert 2 * nsp == W and p.info()["interp_coil_group"] == cg
    gen = torch.Generator(device="cuda").manual_seed(1)
    g = torch.randn((nt * nc,) + tuple(nf), generator=gen, dtype=torch.complex64, device="cuda")
    k = p.interp(g).cpu().numpy()
    for q in sorted({0, nt - 1}):
        take = np.arange(off[q], off[q + 1])[:: max(1, (off[q + 1] - off[q]) // 1500)]
        ref = np.prod(nf) * O.interp(tuple(v[take] for v in xs), g[q * nc:(q + 1) * nc].cpu().numpy(), tau, nsp).T
        assert rel(k[take], ref) < 2e-5
    p.close()


@pytest.mark.parametrize("W,nc,M", [(8, 2, 8000), (8, 2, 9000), (6, 2, 9000), (10, 2, 9000), (12, 4, 3000), (8, 1, 9000),
                                    (6, 3, 3000)])
def test_gradient_groups(W, nc, M):
    rng = np.random.default_rng(W * nc)
    shape = (20, 20, 20)
    xs = [torch.from_numpy(v).cuda() for v in rng.uniform(-np.pi, np.pi, (3, M))]
    gen = torch.Generator(device="cuda").manual_seed(1)
    y = torch.randn(M, nc, generator=gen, dtype=torch.complex64, device="cuda")
    out = []
    for cg in (0, 1, 2):
        p = NufftPlan(3, shape, n_coil=nc, eps=EPS[W], tuning=Tuning(interp_coil_group=cg)).set_points(xs)
        g = torch.randn(p.grid().shape, generator=torch.Generator(device="cuda").manual_seed(2), dtype=torch.complex64,
                        device="cuda")
        out.append(p.interp_grad_coords(g, y).cpu().numpy())
        p.close()
    assert rel(out[0], out[1]) < 1e-5 and rel(out[0], out[2]) < 1e-5
