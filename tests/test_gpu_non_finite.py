"""Values that are not finite reach exactly their own stencil, also on grids of unequal axes,
where weights inside the stencil are below the smallest FP32 number (the Gaussian's width follows
the first axis): the spreads and interps of few coils and of wide stencils.

A sample's stencil is worked out here from its coordinate: n = floor(x / h) in [0, 2 pi), taps
n + 1 - nspread ... n + nspread, periodic.  The sets of cells and samples are compared exactly.
"""
import numpy as np
import pytest
import torch

import oracle as O
from mripy_gb300.plan import NufftPlan, Tuning

pytestmark = pytest.mark.gpu


def stencils(xs, nf, nsp):
    """Boolean (M, *nf): the cells of every sample's stencil."""
    out = None
    for x, n in zip(xs, nf):
        first = np.floor(np.mod(x, 2 * np.pi) / (2 * np.pi / n)).astype(int) + 1 - nsp
        ax = np.zeros((len(x), n), bool)
        for k in range(2 * nsp):
            ax[np.arange(len(x)), (first + k) % n] = True
        out = ax if out is None else out[..., None] & ax.reshape(ax.shape[:1] + (1,) * (out.ndim - 1) + ax.shape[1:])
    return out


@pytest.mark.parametrize("shape,eps,nc,interp_tile", [
    ((40, 20), 1e-15, 1, (0, 0)), ((60, 20), 1e-15, 2, (0, 0)),                    # wide stencils
    ((60, 20), 5e-6, 1, (0, 0)), ((60, 20), 5e-6, 3, (0, 0)),                      # few coils, 2-D spread
    ((48, 32, 16), 5e-6, 1, (0, 0, 0)), ((48, 16, 16), 5e-6, 3, (0, 0, 0)),        # few coils, 3-D: sparse bins,
    ((36, 24, 12), 5e-6, 2, (24, 12, 12)), ((33, 11, 12), 1e-5, 1, (22, 11, 12)),  # and staged windows
    ((36, 12, 12), 1e-6, 1, (12, 12, 12)), ((48, 40, 36), 5e-6, 1, (0, 0, 0))])
def test_values_reach_their_stencil(shape, eps, nc, interp_tile):
    rng = np.random.default_rng(shape[0] + nc)
    dim, M = len(shape), 1000 if min(shape) <= 12 else 400
    nsp, nf, tau = O.grid_params(dim, *shape, eps=eps)
    xs = rng.uniform(-np.pi, np.pi, (dim, M))
    inside = stencils(xs, nf, nsp)
    p = NufftPlan(dim, shape, n_coil=nc, eps=eps, tuning=Tuning(interp_tile=interp_tile))
    p.set_points([torch.from_numpy(v).cuda() for v in xs])
    gen = torch.Generator(device="cuda").manual_seed(1)
    c = torch.randn(M, nc, generator=gen, dtype=torch.complex64, device="cuda")
    g = torch.randn(p.grid().shape, generator=gen, dtype=torch.complex64, device="cuda")
    k0 = p.interp(g).cpu().numpy()
    for value in (float("nan"), float("inf")):
        b = c.clone()
        b[[5, 77]] = complex(value, 1.0)
        got = ~np.isfinite(p.spread(b).cpu().numpy())
        for i in range(nc):
            assert np.array_equal(got[i], inside[5] | inside[77])
        for s in (5, 77):
            cells = np.argwhere(inside[s])
            for cell in (cells[0], cells[-1], cells[len(cells) // 2]):  # two corners and the middle
                h = g.clone()
                h[(slice(None),) + tuple(cell)] = complex(value, 1.0)
                k1 = p.interp(h).cpu().numpy()
                hit = inside[(slice(None),) + tuple(cell)]
                assert np.array_equal(~np.isfinite(k1), np.repeat(hit[:, None], nc, 1))
                assert np.array_equal(k1[~hit], k0[~hit])
    p.close()
