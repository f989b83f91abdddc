"""2-D gridding with wide stencils of more coils than a grid of blocks has rows (65,535): the
wide-stencil kernels take a coil per block and run several launches.

Tolerance: 2e-5 relative L2 (FP32 against the FP64 oracle), as for the other gridding kernels.
"""
import numpy as np
import pytest
import torch

import oracle as O
from mripy_gb300.plan import NufftPlan

pytestmark = pytest.mark.gpu


def test_wide_more_coils_than_grid_rows():
    rng = np.random.default_rng(0)
    nc, M, shape = 65540, 40, (20, 20)
    xs = rng.uniform(-np.pi, np.pi, (2, M))
    p = NufftPlan(2, shape, n_coil=nc).set_points([torch.from_numpy(v).cuda() for v in xs])
    nsp, nf, tau = O.grid_params(2, *shape, eps=1e-15)
    assert p.info()["nspread"] == nsp == 14 and p.info()["spread_tile"] == (32, 32)
    gen = torch.Generator(device="cuda").manual_seed(0)
    c = torch.randn(M, nc, generator=gen, dtype=torch.complex64, device="cuda")
    g = p.spread(c).clone()
    out = p.interp(g).cpu().numpy()
    pick = [0, 1, 32767, 65534, 65535, 65536, nc - 1]
    gp = g.view(nc, *nf)[pick].cpu().numpy()
    ref = O.spread(tuple(xs), c[:, pick].cpu().numpy().T.astype(np.complex128), tau, nsp, nf)
    k = np.prod(nf) * O.interp(tuple(xs), gp, tau, nsp).T
    for i in range(len(pick)):
        assert np.linalg.norm(gp[i] - ref[i]) < 2e-5 * np.linalg.norm(ref[i])
        assert np.linalg.norm(out[:, pick[i]] - k[:, i]) < 2e-5 * np.linalg.norm(k[:, i])
    p.close()
