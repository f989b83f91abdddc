"""The work this framework is used for, as measurable cases.

Each case is one call (or one step) that a reconstruction program makes: the drop-in function
API on a new trajectory, a plan kept for one trajectory, ragged dynamic frames, a
differentiable step, 3-D radial transforms, density compensation and whole solves.  Sizes
follow the benchmark configurations (``mripy_gb300/synth.py``) and the tests; ``draw`` spreads
them over the ranges that those configurations stand for.

``prepare`` makes what a program holds before the call (k-space data, images, coil maps,
trajectory, and the plan or operator where one is kept), ``run`` makes the call, ``work``
counts what the call cannot do without, and ``exact`` evaluates the same result in 64 bits
with direct sums (plain torch), where that takes seconds.
"""
import math

import numpy as np
import torch

from mripy_gb300 import nufft_func, operators, solvers
from mripy_gb300.autograd import nufft_forward
from mripy_gb300.plan import NufftPlan

GOLDEN = math.pi * (math.sqrt(5.0) - 1.0) / 2.0

# kernel widths: eps 5e-6 gives 12 taps per axis (the benchmark's accuracy), the operator
# classes' 1e-5 gives 10, the functions' default 1e-15 gives 28 on a 3x grid
# (12 in 3-D, where the functions clamp the width)
EPS_BENCH, EPS_OPERATOR, EPS_DEFAULT = 5e-6, 1e-5, 1e-15


def listed():
    return [
        # one adjoint through the function API on a new trajectory: the smallest call, a
        # gridding reconstruction of one 128^2 slice (bin sort included, as in every such call)
        dict(name="function_2d_adjoint", kind="function1", dim=2, n=128, aspect=1.0, coils=1, spokes=128, read=256,
             eps=EPS_BENCH),
        # the normal operator through the function API at its default accuracy (eps=1e-15)
        dict(name="function_2d_normal_default", kind="function21", dim=2, n=128, aspect=1.0, coils=1, spokes=128,
             read=256, eps=EPS_DEFAULT),
        # one 3-D forward transform through the function API at its default accuracy
        dict(name="function_3d_forward_default", kind="function2", dim=3, n=64, aspect=1.0, coils=1, spokes=4000,
             read=64, eps=EPS_DEFAULT),
        # a kept 2-D plan, forward then adjoint over the coils of a golden-angle radial scan
        dict(name="plan_2d_8coil", kind="plan", dim=2, n=256, aspect=1.0, coils=8, spokes=402, read=512,
             eps=EPS_BENCH),
        # dynamic series: every frame has its own few spokes, all frames and coils in one plan
        dict(name="frames_2d_12coil", kind="frames", dim=2, n=192, aspect=1.0, coils=12, frames=64, spokes=34,
             read=384, eps=EPS_BENCH),
        # learning the trajectory: forward on new coordinates, gradients of image and coordinates
        dict(name="spiral_gradients_16coil", kind="gradients", dim=2, n=256, aspect=1.0, coils=16, spokes=24,
             read=2048, eps=EPS_BENCH),
        # 3-D radial UTE, 8 coils: the two directions of the largest configuration
        dict(name="ute_3d_forward_8coil", kind="plan2", dim=3, n=128, aspect=1.0, coils=8, spokes=20000, read=128,
             eps=EPS_BENCH),
        dict(name="ute_3d_adjoint_8coil", kind="plan1", dim=3, n=128, aspect=1.0, coils=8, spokes=20000, read=128,
             eps=EPS_BENCH),
        # the SENSE normal operator on an anisotropic matrix with a coil count that is no power of two
        dict(name="sense_3d_normal_12coil", kind="sense", dim=3, n=96, aspect=0.84, coils=12, spokes=6000, read=96,
             eps=EPS_OPERATOR),
        # few-coil 3-D operator, forward then dcf-weighted adjoint
        dict(name="operator_3d_3coil", kind="operator", dim=3, n=72, aspect=1.0, coils=3, spokes=4001, read=73,
             eps=EPS_OPERATOR),
        # density compensation of a 3-D trajectory before its reconstruction (single-coil gridding both ways)
        dict(name="density_3d", kind="density", dim=3, n=96, aspect=1.0, coils=1, spokes=8000, read=96,
             eps=EPS_OPERATOR),
        # a whole wavelet-regularised SENSE reconstruction: 20 FISTA iterations
        dict(name="fista_2d_8coil", kind="fista", dim=2, n=192, aspect=1.0, coils=8, spokes=150, read=384,
             eps=EPS_OPERATOR, iters=20),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["function1", "function21", "function2", "plan", "frames", "gradients", "plan2", "plan1", "sense",
                       "operator", "density", "fista"])
    c = dict(kind=kind, dim=2, aspect=rng.choice([1.0, 1.0, rng.uniform(0.75, 1.0)]), coils=1, eps=EPS_BENCH)
    if kind == "function1":
        c.update(n=_log(rng, 48, 320), coils=rng.choice([1, 1, 2, 4]), eps=rng.choice([EPS_BENCH, EPS_OPERATOR]))
        c.update(spokes=_log(rng, 32, 512), read=2 * c["n"])
    elif kind == "function21":
        c.update(n=_log(rng, 40, 200), coils=rng.choice([1, 1, 2, 3]), eps=EPS_DEFAULT)
        c.update(spokes=_log(rng, 24, 300), read=2 * c["n"])
    elif kind == "function2":
        c.update(dim=3, n=_log(rng, 24, 80), eps=EPS_DEFAULT)
        c.update(spokes=_log(rng, 500, 6000), read=c["n"])
    elif kind == "plan":
        c.update(n=_log(rng, 64, 384), coils=rng.choice([1, 4, 6, 8, 12, 16]))
        c.update(spokes=_log(rng, 48, 600), read=2 * c["n"])
    elif kind == "frames":
        c.update(n=_log(rng, 96, 224), coils=rng.choice([4, 8, 9, 12]), frames=rng.randint(5, 48))
        c.update(spokes=rng.randint(8, 34), read=2 * c["n"])
    elif kind == "gradients":
        c.update(n=_log(rng, 96, 288), coils=rng.choice([1, 4, 8, 12, 16]))
        c.update(spokes=rng.randint(8, 32), read=_log(rng, 512, 2500))
    elif kind in ("plan1", "plan2"):
        c.update(dim=3, n=_log(rng, 40, 128), coils=8)
        c.update(spokes=_log(rng, 2000, 20000), read=c["n"])
    elif kind == "sense":
        c.update(dim=3, n=_log(rng, 32, 104), coils=rng.choice([8, 10, 12, 16]), eps=EPS_OPERATOR)
        c.update(spokes=_log(rng, 1000, 6000), read=c["n"])
    elif kind == "operator":
        c.update(dim=3, n=_log(rng, 32, 96), coils=rng.choice([1, 2, 3, 4, 6]), eps=EPS_OPERATOR)
        c.update(spokes=_log(rng, 1000, 8000), read=c["n"])
    elif kind == "density":
        c.update(dim=3, n=_log(rng, 40, 128), eps=EPS_OPERATOR)
        c.update(spokes=_log(rng, 2000, 12000), read=c["n"])
    else:
        c.update(n=16 * rng.randint(6, 18), coils=rng.choice([4, 8, 12]), eps=EPS_OPERATOR, iters=rng.choice([10, 20]))
        c.update(spokes=_log(rng, 100, 402), read=2 * c["n"])
    if kind == "fista":
        c["aspect"] = 1.0  # the level-4 Haar transform takes sizes that are multiples of 16
    return c


# ---------------------------------------------------------------- inputs

def _shape(c):
    """The first axis is the longest (the kernel's width follows it)."""
    rest = max(8, int(round(c["n"] * c["aspect"])))
    return (c["n"],) + (rest,) * (c["dim"] - 1)


def _rand(gen, *shape):
    return torch.randn(shape, generator=gen, dtype=torch.float32, device="cuda")


def _crand(gen, *shape):
    return torch.complex(_rand(gen, *shape), _rand(gen, *shape))


def _radial_2d(spokes, read, start):
    """Golden-angle spokes through the centre, radians."""
    a = GOLDEN * (start + torch.arange(spokes, dtype=torch.float64, device="cuda"))
    r = 2 * math.pi * (torch.arange(read, dtype=torch.float64, device="cuda") - read / 2.0) / read
    return (torch.cos(a)[:, None] * r).reshape(-1), (torch.sin(a)[:, None] * r).reshape(-1)


def _radial_3d(spokes, read, start):
    """Centre-out spokes on a Fibonacci sphere turned about z by ``start``, radians."""
    i = torch.arange(spokes, dtype=torch.float64, device="cuda") + 0.5
    z = 1.0 - 2.0 * i / spokes
    phi = math.pi * (3.0 - math.sqrt(5.0)) * i + start
    rho = torch.sqrt(1.0 - z * z)
    r = math.pi * torch.arange(read, dtype=torch.float64, device="cuda") / read
    return tuple((d[:, None] * r).reshape(-1) for d in (rho * torch.cos(phi), rho * torch.sin(phi), z))


def _spiral(interleaves, read, gen):
    """Variable-density spiral with perturbed float32 coordinates (2, M), radians."""
    t = torch.arange(read, dtype=torch.float64, device="cuda") / read
    r = 2 * math.pi * 0.4999 * t ** 2
    th = 2 * math.pi * 16 * t
    a = 2 * math.pi * torch.arange(interleaves, dtype=torch.float64, device="cuda") / interleaves
    k = torch.stack([(r * torch.cos(th + a[:, None])).reshape(-1), (r * torch.sin(th + a[:, None])).reshape(-1)])
    return (k + 2e-3 * math.pi * _rand(gen, *k.shape)).to(torch.float32)


def _image(c, gen, coils):
    """A piecewise-smooth object with phase and noise over the given coils, (*shape, coils)."""
    shape = _shape(c)
    ax = torch.meshgrid(*[torch.linspace(-1, 1, s, device="cuda") for s in shape], indexing="ij")
    im = torch.zeros(shape, device="cuda")
    for _ in range(6):
        p = torch.rand(2 * len(shape) + 1, generator=gen, device="cuda")
        d = sum(((a - 0.8 * (p[2 * i] - 0.5)) / (0.15 + 0.6 * p[2 * i + 1])) ** 2 for i, a in enumerate(ax))
        im += (p[-1] - 0.2) * (d <= 1.0)
    ph = _rand(gen, len(shape))
    z = im * torch.exp(1j * sum(ph[i] * a for i, a in enumerate(ax)))
    return z[..., None] * _maps(c, gen, coils) + 0.02 * _crand(gen, *shape, coils)


def _maps(c, gen, coils):
    """Smooth coil maps, sum of squares 1."""
    shape = _shape(c)
    ax = torch.meshgrid(*[torch.linspace(-1, 1, s, device="cuda") for s in shape], indexing="ij")
    out = []
    for k in range(coils):
        ctr = 1.2 * _rand(gen, len(shape))
        f = _rand(gen, len(shape))
        d2 = sum((a - ctr[i]) ** 2 for i, a in enumerate(ax))
        out.append(torch.exp(-d2 / 1.5) * torch.exp(1j * sum(f[i] * a for i, a in enumerate(ax))))
    s = torch.stack(out, dim=-1)
    return s / torch.sqrt((s.abs() ** 2).sum(-1, keepdim=True) + 1e-12)


def _kdata(coords, coils, gen):
    """Samples whose magnitude falls off from the k-space centre as an object's does."""
    r = torch.sqrt(sum(k.double() ** 2 for k in coords)).float()
    return (1.0 / (0.02 + (r / math.pi) ** 1.5))[:, None] * _crand(gen, r.numel(), coils)


def _ramp(coords):
    r = torch.sqrt(sum(k.double() ** 2 for k in coords))
    return ((r / math.pi) ** (len(coords) - 1) + 1e-3).float()


def _frame_spokes(c):
    """Uneven spoke counts of a series' frames, 5 up to the case's (part of the sizes, not of the inputs)."""
    return np.random.default_rng(c["frames"]).integers(min(5, c["spokes"]), c["spokes"] + 1, c["frames"]).tolist()


def _inputs(c, seed):
    """Everything the call reads, from the seed alone."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    kind, d = c["kind"], {}
    turn = int(torch.randint(1, 1000, (1,), generator=gen, device="cuda"))
    if kind == "gradients":
        d["k"] = _spiral(c["spokes"], c["read"], gen)
        d["x"] = _image(c, gen, c["coils"])[None]
        d["g"] = _kdata(d["k"], c["coils"], gen)
        return d
    if kind == "frames":
        per = _frame_spokes(c)
        ks, off = [], [0]
        for s in per:
            ks.append(_radial_2d(s, c["read"], turn))
            turn += s
            off.append(off[-1] + s * c["read"])
        d["k"], d["off"] = tuple(torch.cat([k[i] for k in ks]) for i in range(2)), off
        base = _image(c, gen, c["coils"])
        d["x"] = base[None] + 0.1 * _crand(gen, c["frames"], *base.shape)
        d["y"] = _kdata(d["k"], c["coils"], gen)
        return d
    d["k"] = (_radial_2d if c["dim"] == 2 else _radial_3d)(c["spokes"], c["read"], turn)
    if kind in ("function21", "function2", "plan", "plan2", "operator"):
        d["x"] = _image(c, gen, c["coils"])
    if kind in ("function1", "plan", "plan1", "operator", "fista"):
        d["y"] = _kdata(d["k"], c["coils"], gen)
    if kind in ("sense", "operator"):
        d["dcf"] = _ramp(d["k"])
    if kind in ("sense", "fista"):
        d["s"] = _maps(c, gen, c["coils"])
    if kind == "sense":
        d["x"] = _image(c, gen, 1)[..., 0]
    return d


def _step_threshold(c):
    """A radial scan samples the k-space centre about n times the mean density, which bounds
    the normal operator; the threshold is a hundredth of the first step's image."""
    return 0.5 / c["n"], 0.005 / c["n"]


def prepare(case, seed):
    c = case
    d = _inputs(c, seed)
    kind, shape = c["kind"], _shape(c)
    d["case"] = c
    if kind in ("plan", "plan1", "plan2"):
        d["plan"] = NufftPlan(c["dim"], shape, n_coil=c["coils"], eps=c["eps"]).set_points(list(d["k"]))
    elif kind == "frames":
        d["plan"] = NufftPlan(2, shape, n_coil=c["coils"], n_traj=c["frames"], eps=c["eps"])
        d["plan"].set_points(list(d["k"]), traj_offsets=d["off"])
    elif kind == "gradients":
        d["plan"] = NufftPlan(2, shape, n_coil=c["coils"], eps=c["eps"])
    elif kind == "density":
        d["op"] = operators.NUFFT3d(shape, None, *d["k"])
        d["op"].plan(1)
    elif kind in ("sense", "operator"):
        d["op"] = operators.NUFFT3d(shape, d["dcf"], *d["k"])
        d["op"].plan(c["coils"])
    elif kind == "fista":
        d["op"] = operators.NUFFT2d(shape, None, *d["k"])
        d["op"].plan(c["coils"])
    if kind in ("sense", "fista"):
        d["op"] = operators.joint2operators(operators.espirit(d["s"]), d["op"])
    if kind == "fista":
        d["T"] = solvers.DWTnd("haar", 4, axes=(0, 1))
        # data scaled so that the adjoint image has unit size, as the step and threshold assume
        d["y"] = d["y"] / d["op"].backward(d["y"]).abs().max()
    return d


def run(state):
    d, c = state, state["case"]
    kind, shape = c["kind"], _shape(c)
    if kind == "function1":
        return nufft_func.nufft2d1_gaussker(*d["k"], d["y"], *shape, eps=c["eps"])
    if kind == "function21":
        return nufft_func.nufft2d21_gaussker(*d["k"], d["x"], *shape)
    if kind == "function2":
        return nufft_func.nufft3d2_gaussker(*d["k"], d["x"], *shape)
    if kind == "plan":
        return d["plan"].type2(d["x"][None]), d["plan"].type1(d["y"])
    if kind == "frames":
        return d["plan"].type2(d["x"]), d["plan"].type1(d["y"])
    if kind == "plan2":
        return d["plan"].type2(d["x"][None])
    if kind == "plan1":
        return d["plan"].type1(d["y"])
    if kind == "gradients":
        x, k = d["x"].detach().requires_grad_(), d["k"].detach().requires_grad_()
        out = nufft_forward(x, k, d["plan"])
        gx, gk = torch.autograd.grad(out, (x, k), d["g"])
        return out.detach(), gx, gk
    if kind == "sense":
        return d["op"].forward_backward(d["x"])
    if kind == "operator":
        return d["op"].forward(d["x"]), d["op"].backward(d["y"])
    if kind == "density":
        return d["op"].pipe_menon_dcf(20)
    return solvers.FIST_wrap(d["op"], d["T"], d["y"], c["iters"], *_step_threshold(c))


# ---------------------------------------------------------------- what a pass cannot do without

def _taps(c):
    rat = 2 if c["eps"] > 1e-11 else 3
    ns = int(-math.log(c["eps"]) / (math.pi * (rat - 1) / (rat - 0.5)) + 0.5)
    if c["dim"] == 3 and c["kind"] not in ("plan", "plan1", "plan2"):
        ns = max(3, min(ns, 6))
    return 2 * ns, rat


def _samples(c):
    return float(c["read"] * (sum(_frame_spokes(c)) if c["kind"] == "frames" else c["spokes"]))


def work(case):
    c = case
    W, rat = _taps(c)
    M, nc, fr, kind = _samples(c), c["coils"], c.get("frames", 1), c["kind"]
    pix = fr * float(np.prod(_shape(c)))
    cells = pix * rat ** c["dim"]
    coords, img, smp = 8.0 * c["dim"] * M, 8.0 * pix * nc, 8.0 * M * nc
    grid = 4.0 * W ** c["dim"] * M * nc                     # the stencil's multiply-adds, one direction
    fft = 5.0 * cells * nc * math.log2(cells / fr)          # one transform of the oversampled grids
    one = grid + fft
    table = {
        "function1": (coords + smp + img, one),
        "function2": (coords + smp + img, one),
        "function21": (coords + 2 * img, 2 * one),
        "plan1": (coords + smp + img, one),
        "plan2": (coords + smp + img, one),
        "plan": (coords + 2 * smp + 2 * img, 2 * one),
        "frames": (coords + 2 * smp + 2 * img, 2 * one),
        "operator": (coords + 2 * smp + 2 * img + 4 * M, 2 * one),
        "gradients": (2 * coords / 2 + 2 * smp + 2 * img, 2 * one + grid * (1 + c["dim"])),
        "sense": (coords + img + 16 * pix + 4 * M, 2 * one),
        "density": (coords + 4 * M, 20 * 2 * grid / 2),     # the weights are real
        "fista": (coords + smp + img + 8 * pix, (2 * c.get("iters", 0) + 1) * one),
    }
    b, f = table[kind]
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------- the same results in 64 bits

def _phases(k, n):
    j = torch.arange(-(n // 2), n - n // 2, dtype=torch.float64, device="cuda")
    a = k.double()[:, None] * j
    return torch.complex(torch.cos(a), torch.sin(a))


_CHUNK = 1 << 15  # samples at a time


def _chunks(k):
    for s in range(0, k[0].numel(), _CHUNK):
        yield slice(s, min(s + _CHUNK, k[0].numel()))


def _direct2(k, x, deriv=None):
    """sum_n x_n exp(-i k.n), x (*shape, coils) -> (M, coils); deriv: d/dk of that axis."""
    shape, nc = x.shape[:-1], x.shape[-1]
    x = x.to(torch.complex128)
    if deriv is not None:
        n = shape[deriv]
        j = torch.arange(-(n // 2), n - n // 2, dtype=torch.float64, device="cuda")
        x = x * (-1j * j).reshape([-1 if a == deriv else 1 for a in range(len(shape))] + [1])
    out = torch.empty((k[0].numel(), nc), dtype=torch.complex128, device="cuda")
    for sl in _chunks(k):
        e = [_phases(k[a][sl], shape[a]).conj() for a in range(len(shape))]
        step = max(1, (1 << 27) // (e[0].shape[0] * int(np.prod(shape[1:-1], initial=1)) * nc))
        part = 0
        for i in range(0, shape[0], step):  # bounds the first contraction's size
            xi = x[i:i + step]
            t = torch.einsum("mz,zq->mq", e[-1], xi.movedim(-2, 0).reshape(shape[-1], -1))
            t = t.reshape((-1,) + tuple(xi.shape[:-2]) + (nc,))
            if len(shape) == 3:
                t = torch.einsum("my,mxyc->mxc", e[1], t)
            part = part + torch.einsum("mx,mxc->mc", e[0][:, i:i + step], t)
        out[sl] = part
    return out


def _direct1(k, y, shape):
    """sum_m y_m exp(+i k.n), y (M, coils) -> (*shape, coils)."""
    nc = y.shape[-1]
    y = y.to(torch.complex128)
    out = torch.zeros(tuple(shape) + (nc,), dtype=torch.complex128, device="cuda")
    for sl in _chunks(k):
        e = [_phases(k[a][sl], shape[a]) for a in range(len(shape))]
        step = max(1, (1 << 27) // (e[0].shape[0] * int(np.prod(shape[1:-1], initial=1)) * nc))
        for i in range(0, shape[0], step):
            t = torch.einsum("mx,mc->mxc", e[0][:, i:i + step], y[sl])
            if len(shape) == 3:
                t = torch.einsum("my,mxc->mxyc", e[1], t)
            q = torch.einsum("mz,mq->zq", e[-1], t.reshape(t.shape[0], -1))
            out[i:i + step] += q.reshape((shape[-1],) + tuple(t.shape[1:])).movedim(0, -2)
    return out


def _gridding(k, shape, W, rat):
    """The Gaussian-gridding kernel's pieces in 64 bits: first cells and weights per axis."""
    tau = math.pi * (W / 2 / (rat * (rat - 0.5))) / shape[0] ** 2
    cells, weights, nf = [], [], []
    for a in range(len(shape)):
        n = max(rat * shape[a], W)
        h = 2 * math.pi / n
        u = torch.remainder(k[a].double(), 2 * math.pi) / h
        first = torch.floor(u) - (W // 2 - 1)
        j = torch.arange(W, dtype=torch.float64, device="cuda")
        d = (u - first)[:, None] - j
        weights.append(torch.exp(-(d * h) ** 2 / (4 * tau)))
        cells.append(torch.remainder(first[:, None] + j, n).long())
        nf.append(n)
    return cells, weights, nf


def _density(c, k, iters=20):
    W, rat = _taps(c)
    cells, w, nf = _gridding(k, _shape(c), W, rat)
    M = k[0].numel()
    dens = torch.ones(M, dtype=torch.float64, device="cuda")
    yz = ((cells[1] * nf[2])[:, :, None] + cells[2][:, None, :]).reshape(M, -1)
    wyz = (w[1][:, :, None] * w[2][:, None, :]).reshape(M, -1)
    for _ in range(iters):
        g = torch.zeros(int(np.prod(nf)), dtype=torch.float64, device="cuda")
        for t in range(W):
            i = cells[0][:, t:t + 1] * (nf[1] * nf[2]) + yz
            g.index_add_(0, i.reshape(-1), ((dens * w[0][:, t])[:, None] * wyz).reshape(-1))
        back = torch.zeros_like(dens)
        for t in range(W):
            i = cells[0][:, t:t + 1] * (nf[1] * nf[2]) + yz
            back += w[0][:, t] * (g[i] * wyz).sum(1)
        dens = dens / back.abs()
    return dens * M / dens.sum()


def _haar(x, level, inverse):
    """Orthonormal Haar transform over the two image axes, approximation block first."""
    x = x.clone()
    for lv in (reversed(range(level)) if inverse else range(level)):
        n = [s >> lv for s in x.shape[:2]]
        b = x[:n[0], :n[1]]
        for a in (0, 1):
            if inverse:
                lo, hi = b.split(n[a] // 2, dim=a)
                b = torch.stack([lo + hi, lo - hi], dim=a + 1).reshape(b.shape) / math.sqrt(2.0)
            else:
                p = b.unflatten(a, (n[a] // 2, 2))
                lo, hi = p.select(a + 1, 0), p.select(a + 1, 1)
                b = torch.cat([lo + hi, lo - hi], dim=a) / math.sqrt(2.0)
        x[:n[0], :n[1]] = b
    return x


def _fista(k, s, y, shape, iters, step, th):
    M = k[0].numel()
    e = [_phases(k[a], shape[a]) for a in range(2)]
    s = s.to(torch.complex128)

    def normal(x):
        t = x[..., None] * s                                     # (n0, n1, c)
        f = torch.einsum("my,xyc->mxc", e[1].conj(), t)
        f = torch.einsum("mx,mxc->mc", e[0].conj(), f)
        return adjoint(f)

    def adjoint(f):
        t = torch.einsum("mx,mc->mxc", e[0], f).reshape(M, -1)
        g = (e[1].T @ t).reshape(shape[1], shape[0], -1).movedim(0, 1)
        return (g * s.conj()).sum(-1) / M

    rhs = adjoint(y.to(torch.complex128))
    v, t0 = step * rhs, 1.0
    acc, prev = torch.zeros_like(v), v
    x = v
    for _ in range(iters):
        acc = acc - step * (normal(v) - rhs)
        q = _haar(acc, 4, False)
        a = q.abs()
        x = _haar(q / (a + 1e-6) * torch.clamp(a - th, min=0.0), 4, True)
        t1 = (1 + math.sqrt(1 + 4 * t0 * t0)) / 2
        v, prev, t0 = x + ((t0 - 1) / t1) * (x - prev), x, t1
    return x


def _cost(c):
    """Complex 64-bit operations (eight flops each) of the direct sums of one pass, roughly."""
    one = _samples(c) * float(np.prod(_shape(c))) * c["coils"]
    passes = {"function21": 2, "plan": 2, "frames": 2, "gradients": 4, "sense": 2, "operator": 2,
              "fista": 2 * c.get("iters", 0) + 1}.get(c["kind"], 1)
    return 8.0 * one * passes


def exact(case, seed):
    c, kind, shape = case, case["kind"], _shape(case)
    if kind == "density":
        if 40.0 * _taps(c)[0] ** 3 * _samples(c) > 4e10:
            return None
    elif _cost(c) > 6e12:
        return None
    d = _inputs(c, seed)
    k = d["k"]
    if kind in ("function1", "plan1"):
        out = _direct1(k, d["y"], shape) / k[0].numel()
        return out if kind == "function1" else out[None]
    if kind in ("function2", "plan2"):
        return _direct2(k, d["x"])
    if kind == "function21":
        return _direct1(k, _direct2(k, d["x"]), shape) / k[0].numel()
    if kind == "plan":
        return _direct2(k, d["x"]), _direct1(k, d["y"], shape)[None] / k[0].numel()
    if kind == "frames":
        out, im, off = [], [], d["off"]
        for f in range(c["frames"]):
            kf = tuple(a[off[f]:off[f + 1]] for a in k)
            out.append(_direct2(kf, d["x"][f]))
            im.append(_direct1(kf, d["y"][off[f]:off[f + 1]], shape) / (off[f + 1] - off[f]))
        return torch.cat(out), torch.stack(im)
    if kind == "gradients":
        g = d["g"].to(torch.complex128)
        gk = torch.stack([(g.conj() * _direct2(k, d["x"][0], deriv=a)).sum(1).real for a in range(2)])
        return _direct2(k, d["x"][0]), _direct1(k, d["g"], shape)[None], gk
    if kind == "sense":
        s = d["s"].to(torch.complex128)
        f = _direct2(k, d["x"].to(torch.complex128)[..., None] * s) * d["dcf"].double()[:, None]
        return (_direct1(k, f, shape) * s.conj()).sum(-1, keepdim=True) / k[0].numel()
    if kind == "operator":
        return _direct2(k, d["x"]), _direct1(k, d["y"] * d["dcf"].double()[:, None], shape) / k[0].numel()
    if kind == "density":
        return _density(c, k)
    # the data scaled as prepare does, in 64 bits
    e = _direct1(k, d["y"], shape) * d["s"].to(torch.complex128).conj()
    y = d["y"].to(torch.complex128) / (e.sum(-1) / k[0].numel()).abs().max()
    return _fista(k, d["s"], y, shape, c["iters"], *_step_threshold(c))[..., None]
