"""The fused image <-> grid transforms (band_fft.cuh: pad, deapodisation and crop fused with
band-limited FFTs) against the general path (``fft_variant`` 1: pad kernel, cuFFT over the whole
grid, crop kernel) on the same plan geometry.

Covered: every supported grid length in 2-D, mixed lengths in 3-D, odd image sizes, coil counts
that fill a block's 16 lines and that do not (chunks, several rows per block), more than 16
coils, coil-last and coil-major images, strided samples, several groups, both signs of iflag,
the SENSE forms, pinned host images, captured graphs and a length without kernels.

Tolerance.  Two FP32 transforms of N cells each differ from the exact one by about
0.5 eps sqrt(log2 N) in relative L2 (random rounding, eps = 6e-8 per operation, a few operations
a level): 1e-7 to 2e-7 for these grids.  Their difference, with the scaling's roundings, stays
below 1e-6; gridding differences (the order of float atomics) are below 5e-7 more.
"""
import numpy as np
import pytest
import torch

from mripy_gb300 import _native as N
from mripy_gb300.plan import NufftPlan, Tuning

pytestmark = pytest.mark.gpu

TOL = 2e-6
LENGTHS = [64, 72, 80, 96, 100, 108, 112, 120, 128, 144, 150, 160, 162, 168, 180, 192, 200, 216, 224, 240, 256, 270,
           288, 300, 320, 324, 336, 360, 384, 400, 432, 480, 512, 576, 640, 768]


def rel(a, b):
    return float((a - b).norm() / b.norm())


def crand(gen, *shape):
    return torch.randn(shape, generator=gen, dtype=torch.complex64, device="cuda")


def plans(dim, shape, M, gen, n_coil=1, n_traj=1, eps=1e-5, iflag=1):
    ks = [2 * np.pi * (torch.rand(M, generator=gen, dtype=torch.float64, device="cuda") - 0.5) for _ in range(dim)]
    off = [0] + [M * (g + 1) // n_traj for g in range(n_traj)]
    out = []
    for fv in (0, 1):
        p = NufftPlan(dim, shape, n_coil=n_coil, n_traj=n_traj, eps=eps, iflag=iflag, max_nspread=6 if dim == 3 else None,
                      tuning=Tuning(fft_variant=fv))
        out.append(p.set_points(ks, traj_offsets=off))
    return out


@pytest.mark.parametrize("nf", LENGTHS)
def test_every_length_both_axes(nf):
    gen = torch.Generator(device="cuda").manual_seed(nf)
    own, ref = plans(2, (nf // 2, nf // 2), 700, gen, n_coil=3)
    assert own.info()["nf"] == (nf, nf)
    x, y = crand(gen, 1, nf // 2, nf // 2, 3), crand(gen, 700, 3)
    own.type2(x), ref.type2(x)
    assert rel(own.grid(), ref.grid()) < TOL                    # the transformed grid itself
    assert rel(own.type1(y), ref.type1(y)) < TOL
    # against 64 bits: no further off than the library's transform (within the spread of both)
    g64 = torch.fft.fft2(ref.pad_deapod(x).to(torch.complex128))
    own.type2(x), ref.type2(x)
    assert rel(own.grid().to(torch.complex128), g64) < 4e-7
    own.close(), ref.close()


@pytest.mark.parametrize("dim,shape,eps", [
    (2, (81, 36), 1e-5), (2, (100, 72), 1e-5), (2, (64, 27), 1e-12), (3, (36, 32, 40), 1e-5), (3, (48, 27, 36), 1e-12),
    (3, (75, 36, 32), 1e-5)])
@pytest.mark.parametrize("nc,nt", [(1, 3), (2, 1), (5, 2), (8, 1), (12, 2), (16, 1), (19, 1), (33, 1)])
def test_coils_groups_layouts(dim, shape, eps, nc, nt):
    gen = torch.Generator(device="cuda").manual_seed(7 * nc + nt)
    own, ref = plans(dim, shape, 400, gen, n_coil=nc, n_traj=nt, eps=eps, iflag=1 if nc % 2 else -1)
    x = crand(gen, nt, *shape, nc)
    xm = torch.empty((nt, nc) + shape, dtype=torch.complex64, device="cuda").movedim(1, -1)  # coil-major
    xm.copy_(x)
    y = crand(gen, 400, nc)
    k0 = ref.type2(x)
    assert rel(own.type2(x), k0) < TOL and rel(own.type2(xm), k0) < TOL
    f0 = ref.type1(y)
    out = torch.empty((nt, nc) + shape, dtype=torch.complex64, device="cuda").movedim(1, -1)
    assert rel(own.type1(y), f0) < TOL and rel(own.type1(y, out=out), f0) < TOL
    assert rel(own.type21(x), ref.type21(x)) < 2 * TOL
    s = crand(gen, *shape, nc)
    sm = torch.empty((nc,) + shape, dtype=torch.complex64, device="cuda").movedim(0, -1)
    sm.copy_(s)
    v = crand(gen, nt, *shape)
    for m in (s, sm):
        assert rel(own.sense_forward(v, m), ref.sense_forward(v, s)) < TOL
        assert rel(own.sense_adjoint(y, m), ref.sense_adjoint(y, s)) < TOL
        assert rel(own.sense_normal(v, m), ref.sense_normal(v, s)) < 2 * TOL
    own.close(), ref.close()


def test_host_images_graphs_and_unsupported_lengths():
    gen = torch.Generator(device="cuda").manual_seed(3)
    own, ref = plans(2, (64, 48), 500, gen, n_coil=12)
    x, y = crand(gen, 1, 64, 48, 12), crand(gen, 500, 12)
    lib = N.lib()
    hx, hk = x.cpu().pin_memory(), torch.empty(500, 12, dtype=torch.complex64).pin_memory()
    N.check(lib.gbn_type2_host(own._h, hx.data_ptr(), hk.data_ptr(), None))
    assert rel(hk.cuda(), ref.type2(x)) < TOL
    hy, hf = y.cpu().pin_memory(), torch.empty(1, 64, 48, 12, dtype=torch.complex64).pin_memory()
    N.check(lib.gbn_type1_host(own._h, hy.data_ptr(), hf.data_ptr(), None))
    assert rel(hf.cuda(), ref.type1(y)) < TOL
    out = torch.empty_like(x)
    g = own.capture_normal(x, out)
    g.launch()
    torch.cuda.synchronize()
    assert rel(out, ref.type21(x)) < 2 * TOL
    g.close(), own.close(), ref.close()
    own, ref = plans(2, (64, 47), 500, gen)  # 94 = 2 x 47: the general path
    x = crand(gen, 1, 64, 47, 1)
    assert torch.equal(own.type2(x), ref.type2(x))
    own.close(), ref.close()
