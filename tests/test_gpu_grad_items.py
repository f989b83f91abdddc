"""3-D coordinate gradients whose block takes several work items of a bin: items of 64 and of odd
sizes, bins of one item to dozens, against a plan whose items a block takes whole.

Tolerance: 1e-5 relative L2 (two FP32 sums of the same terms in another order).
"""
import numpy as np
import pytest
import torch

from mripy_gb300.plan import NufftPlan, Tuning

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eps,nc,M", [
    (1e-3, 4, 66000), (1e-3, 6, 44000), (1e-2, 3, 12000), (1e-2, 4, 9000), (1e-2, 2, 70000)])
def test_gradients_over_items(eps, nc, M):
    rng = np.random.default_rng(nc)
    shape = (20, 18, 16)
    xs = rng.uniform(-np.pi, np.pi, (3, M))
    xs[:, : M // 3] *= 0.05
    ks = [torch.from_numpy(v).cuda() for v in xs]
    gen = torch.Generator(device="cuda").manual_seed(1)
    y = torch.randn(M, nc, generator=gen, dtype=torch.complex64, device="cuda")
    out = []
    for tu in (Tuning(interp_coil_group=1), None, Tuning(max_subproblem=40), Tuning(max_subproblem=7, interp_threads=128)):
        p = NufftPlan(3, shape, n_coil=nc, n_traj=2, eps=eps, tuning=tu)
        p.set_points(ks, traj_offsets=[0, M // 2 + 5, M])
        g = torch.randn(p.grid().shape, generator=torch.Generator(device="cuda").manual_seed(2), dtype=torch.complex64,
                        device="cuda")
        out.append(p.interp_grad_coords(g, y).cpu().numpy())
        p.close()
    for o in out[1:]:
        assert np.linalg.norm(o - out[0]) < 1e-5 * np.linalg.norm(out[0])
