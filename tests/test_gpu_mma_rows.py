"""The row order of the 3-D tensor-core kernels' work lists: batches whose samples reach only some
of a tile's y rows (skipped chunks of the interp, zero quarters of the spread), against the FP64
oracle.

Covered: samples in thin y slabs at every offset against the tiles (1 to 4 chunks a batch, one
chunk throughout, chunk counts of both parities across batches), batches that end mid-way,
items of many batches and split tiles' interleaved items, two coil groups, odd grids, and the
plan's other interp on the same lists.  Tolerance 2e-5 relative L2, as for these kernels.
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


def rel(a, b):
    return float(np.linalg.norm(a.cpu().numpy() - b) / np.linalg.norm(b))


@pytest.mark.parametrize("eps,shape", [(1e-3, (24, 26, 22)), (1e-5, (24, 27, 23)), (5e-6, (24, 25, 24)), (1e-7, (26, 26, 26))])
@pytest.mark.parametrize("max_sub", [0, 96, 1000])
@pytest.mark.parametrize("nc", [8, 11])
def test_slabs_against_oracle(eps, shape, max_sub, nc):
    rng = np.random.default_rng(nc + max_sub)
    nsp, nf, tau = O.grid_params(3, *shape, eps=eps)
    xs = []
    for y0 in np.linspace(-np.pi, np.pi, 9):                     # slabs a fraction of a cell thick
        m = int(rng.integers(60, 900))
        x = rng.uniform(-np.pi, np.pi, (3, m))
        x[1] = y0 + rng.uniform(0, 0.3, m) * 2 * np.pi / nf[1]
        x[0, : m // 2] *= 0.1                                    # long items in some tiles
        x[2, : m // 2] *= 0.1
        xs.append(x)
    xs = np.concatenate(xs, axis=1)[:, rng.permutation(sum(x.shape[1] for x in xs))]
    M = xs.shape[1]
    c = (rng.standard_normal((M, nc)) + 1j * rng.standard_normal((M, nc))).astype(np.complex64)
    G = (rng.standard_normal((nc,) + nf) + 1j * rng.standard_normal((nc,) + nf)).astype(np.complex64)
    gref = O.spread(tuple(xs), c.T, tau, nsp, nf)
    cref = np.prod(nf) * O.interp(tuple(xs), G, tau, nsp).T
    for variant in (0, 1):
        p = NufftPlan(3, shape, n_coil=nc, eps=eps, tuning=Tuning(max_subproblem=max_sub, interp_variant=variant))
        p.set_points([cuda(v) for v in xs])
        inf = p.info()
        assert inf["spread_variant"] == 3 and inf["interp_variant"] == (1 if variant else 2)
        assert rel(p.spread(cuda(c)), gref) < TOL_REF
        assert rel(p.interp(cuda(G)), cref) < TOL_REF
        p.status()
        p.close()
