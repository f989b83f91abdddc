"""A call that the library refuses with a CUDA error leaves none behind for the calls after it.

The gradients over bins of 40^3 cells want more shared memory than a block may have, which the host
side is told before any launch.
"""
import numpy as np
import pytest
import torch

from mripy_gb300._native import GbnError
from mripy_gb300.plan import NufftPlan, Tuning

pytestmark = pytest.mark.gpu


def test_refused_call_leaves_no_error():
    rng = np.random.default_rng(0)
    xs = [torch.from_numpy(v).cuda() for v in rng.uniform(-np.pi, np.pi, (3, 500))]
    c = torch.randn(500, 2, dtype=torch.complex64, device="cuda")
    p = NufftPlan(3, (24, 24, 24), eps=1e-6, tuning=Tuning(interp_tile=(40, 40, 40))).set_points(xs)
    g = p.spread(c[:, :1].contiguous())
    with pytest.raises(GbnError):
        p.interp_grad_coords(g, c[:, :1].contiguous())
    q = NufftPlan(3, (24, 24, 24), n_coil=2, eps=1e-6).set_points(xs)  # launches kernels of its own
    q.type1(c)
    with pytest.raises(GbnError):
        p.interp_grad_coords(g, c[:, :1].contiguous())
    p.spread(c[:, :1].contiguous())  # and so does another call of the same plan
    torch.cuda.synchronize()
    q.close()
    p.close()
