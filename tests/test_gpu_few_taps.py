"""The few-coil kernels at their narrowest stencils, 2 and 4 taps per axis: spreads and interps of
1 to 3 coils in 2-D and 3-D, sparse and dense bins, against the FP64 oracle.

Tolerance: 2e-5 relative L2 (FP32 against the FP64 oracle), as for the other gridding kernels.
"""
import numpy as np
import pytest
import torch

import oracle as O
from mripy_gb300.plan import NufftPlan

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("eps,ns", [(0.09, 1), (1e-2, 2)])
@pytest.mark.parametrize("nc", [1, 2, 3])
@pytest.mark.parametrize("shape,M", [((20, 17, 18), 400), ((20, 17, 18), 20000), ((40, 37), 300), ((40, 37), 9000)])
def test_two_and_four_taps(shape, M, nc, eps, ns):
    rng = np.random.default_rng(M + nc)
    dim = len(shape)
    xs = rng.uniform(-np.pi, np.pi, (dim, M))
    xs[:, :M // 4] *= 0.1
    xs[:, -20:] = np.pi
    nsp, nf, tau = O.grid_params(dim, *shape, eps=eps)
    p = NufftPlan(dim, shape, n_coil=nc, eps=eps).set_points([torch.from_numpy(v).cuda() for v in xs])
    assert p.info()["nspread"] == nsp == ns
    assert p.info()["spread_tile"] == ((8, 8, 16 if nc == 1 else 8) if dim == 3 else (32, 32))
    c = (rng.standard_normal((M, nc)) + 1j * rng.standard_normal((M, nc))).astype(np.complex64)
    g = p.spread(torch.from_numpy(c).cuda()).cpu().numpy()
    assert rel(g, O.spread(tuple(xs), c.T, tau, nsp, nf)) < 2e-5
    G = (rng.standard_normal((nc,) + tuple(nf)) + 1j * rng.standard_normal((nc,) + tuple(nf))).astype(np.complex64)
    k = p.interp(torch.from_numpy(G).cuda()).cpu().numpy()
    assert rel(k, np.prod(nf) * O.interp(tuple(xs), G, tau, nsp).T) < 2e-5
    p.close()
