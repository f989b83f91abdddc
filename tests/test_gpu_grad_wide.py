"""Coordinate gradients with stencils above 16 taps, whose samples share a block's idle threads:
items of one sample to full ones, every group of coils, 1-D to 3-D, against central differences of
the FP64 oracle's interp.

Tolerance: 2e-5 relative L2, as for the other gridding kernels (FP32 against FP64).  The differences
are exact to 1e-6: a step of 1e-5 is 4e-4 cells of the finest grid here, its square over six times
the third derivative's ratio to the first (3 at most) 1e-7.
"""
import numpy as np
import pytest
import torch

import oracle as O
from mripy_gb300.plan import NufftPlan, Tuning

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,shape,nc,eps,tuning", [
    (2, (48, 44), 1, 1e-9, None), (2, (48, 44), 2, 1e-15, None), (2, (40, 36), 3, 1e-15, None),
    (2, (48, 44), 8, 1e-12, Tuning(interp_threads=128)), (2, (44, 48), 12, 1e-9, Tuning(max_subproblem=7)),
    (2, (48, 44), 2, 1e-17, None), (1, (300,), 2, 1e-15, None), (3, (24, 22, 20), 1, 1e-9, Tuning(interp_tile=(4, 4, 4)))])
def test_wide_gradients(dim, shape, nc, eps, tuning):
    rng = np.random.default_rng(nc * dim)
    nsp, nf, tau = O.grid_params(dim, *shape, eps=eps)
    assert 2 * nsp > 16
    M = 900
    xs = rng.uniform(-np.pi, np.pi, (dim, M))
    xs[:, :400] *= 0.02  # a bin with several items
    xs[:, 400:440] = 0.3 * np.pi + 0.01 * xs[:, 400:440]  # and one with a partly filled item
    p = NufftPlan(dim, shape, n_coil=nc, eps=eps, tuning=tuning).set_points([torch.from_numpy(v).cuda() for v in xs])
    nf = tuple(nf)[:dim]
    G = (rng.standard_normal((nc,) + nf) + 1j * rng.standard_normal((nc,) + nf)).astype(np.complex64)
    y = (rng.standard_normal((M, nc)) + 1j * rng.standard_normal((M, nc))).astype(np.complex64)
    got = p.interp_grad_coords(torch.from_numpy(G).cuda(), torch.from_numpy(y).cuda()).cpu().numpy()
    h = 1e-5
    for d in range(dim):
        step = np.zeros((dim, 1))
        step[d] = h
        up, dn = (O.interp(tuple(xs + s * step), G.astype(np.complex128), tau, nsp) for s in (1, -1))
        ref = np.prod(nf) * np.sum(np.real(np.conj(y.T) * (up - dn)), axis=0) / (2 * h)
        assert np.linalg.norm(got[:, d] - ref) < 2e-5 * np.linalg.norm(ref)
    p.close()
