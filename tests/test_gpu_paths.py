"""Which kernels run: a plan's info and the launches that the profiler sees, so that the tests of
the fused transforms and of the density compensation's real interp cannot pass on the general
path they are compared with.

Skipped where the profiler records no device activity.
"""
import numpy as np
import pytest
import torch

from mripy_gb300.plan import NufftPlan, Tuning

pytestmark = pytest.mark.gpu

LENGTHS = [64, 72, 80, 96, 100, 108, 112, 120, 128, 144, 150, 160, 162, 168, 180, 192, 200, 216, 224, 240, 256, 270,
           288, 300, 320, 324, 336, 360, 384, 400, 432, 480, 512, 576, 640, 768]


def points(dim, M, seed=0):
    rng = np.random.default_rng(seed)
    return [torch.from_numpy(rng.uniform(-np.pi, np.pi, M)).cuda() for _ in range(dim)]


def launched(call):
    """Names of the kernels that the call launches."""
    call()
    torch.cuda.synchronize()
    for _ in range(3):  # a process' first recording can come back empty
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
            call()
            torch.cuda.synchronize()
        names = [e.name for e in prof.events() if e.device_type == torch.autograd.DeviceType.CUDA]
        if names:
            return names
    pytest.skip("the profiler records no device activity")


def any_of(names, word):
    return any(word in n for n in names)


@pytest.mark.parametrize("nf", LENGTHS)
def test_supported_lengths_take_the_fused_transforms(nf):
    for fv in (0, 1, 2):
        p = NufftPlan(2, (nf // 2, nf // 2), n_coil=2, eps=1e-5, tuning=Tuning(fft_variant=fv))
        assert p.info()["nf"] == (nf, nf) and p.info()["band_fft"] == (1 if fv == 0 else 0)
        p.close()


@pytest.mark.parametrize("shape,eps,fused", [
    ((64, 47), 1e-5, 0), ((47, 64), 1e-5, 0), ((63, 64), 1e-5, 0), ((64, 27), 1e-5, 0), ((81, 36), 1e-5, 1),
    ((36, 32, 40), 1e-5, 1), ((36, 32, 41), 1e-5, 0), ((41, 32, 36), 1e-5, 0), ((36, 41, 32), 1e-5, 0),
    ((48, 36, 32), 1e-12, 1), ((64, 48), 1e-12, 1), ((48, 27, 36), 1e-12, 0), ((64, 27), 1e-12, 0), ((64,), 1e-5, 0)])
def test_every_axis_has_to_be_supported(shape, eps, fused):
    p = NufftPlan(len(shape), shape, eps=eps, max_nspread=6 if len(shape) == 3 else None)
    assert p.info()["band_fft"] == fused
    p.close()


@pytest.mark.parametrize("shape", [(64, 48), (48, 36, 32)])
def test_fused_transforms_of_threefold_grids(shape):
    """Against the full transform; 2e-6 as two FP32 transforms and griddings of these sizes differ."""
    nc, M = 3, 400
    gen = torch.Generator(device="cuda").manual_seed(1)
    y = torch.randn(M, nc, generator=gen, dtype=torch.complex64, device="cuda")
    x = torch.randn(1, *shape, nc, generator=gen, dtype=torch.complex64, device="cuda")
    out = []
    for fv in (0, 1):
        p = NufftPlan(len(shape), shape, n_coil=nc, eps=1e-12, max_nspread=6, tuning=Tuning(fft_variant=fv))
        p.set_points(points(len(shape), M))
        assert p.info()["band_fft"] == 1 - fv and p.info()["nf"] == tuple(3 * n for n in shape)
        out.append((p.type1(y), p.type2(x)))
        p.close()
    for a, b in zip(*out):
        assert float((a - b).norm() / b.norm()) < 2e-6


@pytest.mark.parametrize("shape", [(64, 48), (36, 32, 40)])
@pytest.mark.parametrize("sens", [False, True])
def test_composite_calls_launch_the_fused_transforms(shape, sens):
    nc, M = 3, 500
    for fv in (0, 1):
        p = NufftPlan(len(shape), shape, n_coil=nc, eps=1e-5, tuning=Tuning(fft_variant=fv))
        p.set_points(points(len(shape), M))
        y = torch.randn(M, nc, dtype=torch.complex64, device="cuda")
        x = torch.randn(1, *shape, nc, dtype=torch.complex64, device="cuda")
        s = torch.randn(*shape, nc, dtype=torch.complex64, device="cuda")
        if sens:
            names = launched(lambda: p.sense_normal(x[..., 0].contiguous(), s))
        else:
            names = launched(lambda: (p.type1(y), p.type2(x)))
        for word in ("k_fft_rows_in", "k_fft_cols", "k_fft_rows_sense" if sens else "k_fft_rows_out"):
            assert any_of(names, word) == (fv == 0), (word, names)
        for word in ("k_pad", "k_crop"):
            assert any_of(names, word) == (fv == 1), (word, names)
        p.close()


@pytest.mark.parametrize("shape,eps,M,real", [
    ((24, 22, 20), 1e-3, 30000, True), ((24, 22, 20), 1e-4, 30000, True), ((24, 22, 20), 1e-5, 30000, True),
    ((24, 22, 20), 5e-6, 30000, True),
    ((24, 22, 20), 5e-6, 2000, False),     # few samples a bin
    ((24, 22, 20), 1e-6, 30000, False),    # 14 taps
    ((24, 22, 17), 1e-12, 30000, False)])  # odd grid rows
def test_density_compensation_launches_the_real_interp(shape, eps, M, real):
    p = NufftPlan(3, shape, eps=eps, max_nspread=6 if eps < 1e-8 else None).set_points(points(3, M))
    names = launched(lambda: p.pipe_menon_dcf(1))
    assert any_of(names, "k_interp3d_real") == real
    assert any_of(names, "k_interp3d_one") == (not real)
    assert any_of(names, "k_spread3d_few")
    p.close()
