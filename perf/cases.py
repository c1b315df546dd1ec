"""Workloads of the visibility-space operator chain, each through the package's public entry
points: the calls a lens-modelling program makes, from a 128^2 image with 2e4 visibilities to
1e7 visibilities on a 2048^2 grid.

kinds
  nufft         F^T F of an image: NUFFTOperator forward and adjoint on device tensors
  grid          degridding and gridding of one plan, visibilities kept in plan order
  rows          the same on visibilities in the data's own row order, several channels
  normal        one application of the inversion's normal operator (the matvec of every solver)
  solve         one source inversion, from a zero guess to the requested residual
  deflect       source-plane positions of many image-plane points
  sweep         degridding, gridding and deflection of many lens models of uneven size
  precondition  the learned preconditioner on one residual
  train         loss and gradients of the preconditioner's network on one batch
"""
from __future__ import annotations

import math

import numpy as np
import torch

from lentils_gb300 import synthetic
from lentils_gb300.gridding import GriddingPlan
from lentils_gb300.inversion import SourceInversion
from lentils_gb300.learned import UNet, features
from lentils_gb300.lens_models import (ExternalPotential, GlobalLensModel, InternalMultipoles,
                                       PowerLawEllipsoid)
from lentils_gb300.operators import BilinearLensOperator, NUFFTOperator
from lentils_gb300.spaces import ImageSpace, VisibilitySpace
from lentils_gb300.sweep import BatchedSweep, draw_samples

TWO_PI = 6.28318530718  # the phase constant of the gridding operator
Z_SRC = 2.0
PRIOR = 1e-2  # strength of the gradient prior of the workload inversion


# ------------------------------------------------------------------------------------------------
# The cases
# ------------------------------------------------------------------------------------------------
def listed():
    return [
        # a first look at a small data set, and every iteration of a small imaging loop: launch
        # and latency bound
        {"name": "nufft_128_w6", "kind": "nufft", "nx": 128, "ny": 128, "nvis": 20000, "w": 3,
         "beta": 14.04, "pix": 0.02, "off": 0.0, "dtype": "float32"},
        # a cut-out of odd shape away from the phase centre, the operator's default kernel
        {"name": "nufft_250x187_w8", "kind": "nufft", "nx": 250, "ny": 187, "nvis": 131071,
         "w": 4, "beta": 0.0, "pix": 0.015, "off": 0.13, "dtype": "float32"},
        # the double-precision operator of the refinement residuals
        {"name": "nufft_512_w8_f64", "kind": "nufft", "nx": 512, "ny": 512, "nvis": 2000000,
         "w": 4, "beta": 0.0, "pix": 0.01, "off": 0.0, "dtype": "float64"},
        # the largest single operator: 1e7 visibilities, a tenth of them in dense blobs
        {"name": "grid_2048_w8_1e7", "kind": "grid", "n": 1024, "nvis": 10000000, "w": 4,
         "blobs": 0.1},
        # model visibilities and a dirty grid in the data's own row order, four channels
        {"name": "rows_1024_w8_4ch", "kind": "rows", "n": 512, "nrows": 400000, "nch": 4, "w": 4},
        # the solver's matvec at full size
        {"name": "normal_512_vis", "kind": "normal", "n": 512, "nsrc": 128, "nvis": 2000000,
         "term": "visibilities"},
        # the same with the dirty-beam data term, at a smaller image
        {"name": "normal_256_bcb", "kind": "normal", "n": 256, "nsrc": 96, "nvis": 300000,
         "term": "bcb"},
        # a whole source inversion (windowed flexible CG inside FP64 refinement) with a prior
        # about as strong as the data, as the evidence prefers it
        {"name": "solve_512_vis", "kind": "solve", "n": 512, "nsrc": 128, "nvis": 2000000,
         "strength": 1e4, "tol": 1e-8},
        # ray tracing of the pixel grids of 64 images of 512^2
        {"name": "deflect_64x512", "kind": "deflect", "points": 64 * 512 * 512, "order": 4},
        # lens models of uneven image size and visibility count in one launch
        {"name": "sweep_20", "kind": "sweep", "samples": 20, "layout": 7},
        # the network as the solver applies it: one residual on the 128^2 source grid
        {"name": "precondition_128", "kind": "precondition", "h": 128, "wd": 128},
        # a training batch of the network
        {"name": "train_128_b32", "kind": "train", "h": 128, "wd": 128, "batch": 32},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["nufft", "nufft", "grid", "rows", "normal", "solve", "deflect", "sweep",
                       "precondition", "train"])
    if kind == "nufft":
        f64 = rng.random() < 0.35
        return {"kind": kind, "nx": _log_int(rng, 64, 512), "ny": _log_int(rng, 64, 512),
                "nvis": _log_int(rng, 1e4, 2e6), "w": rng.choice([3, 4]), "beta": 0.0,
                "pix": rng.choice([0.01, 0.015, 0.02]), "off": rng.choice([0.0, 0.13, -0.4]),
                "dtype": "float64" if f64 else "float32"}
    if kind == "grid":
        return {"kind": kind, "n": _log_int(rng, 96, 1024), "nvis": _log_int(rng, 3e4, 8e6),
                "w": rng.choice([2, 3, 4]), "blobs": rng.choice([0.0, 0.1])}
    if kind == "rows":
        return {"kind": kind, "n": _log_int(rng, 96, 768), "nrows": _log_int(rng, 1e4, 5e5),
                "nch": rng.choice([1, 2, 3, 8]), "w": rng.choice([3, 4])}
    if kind == "normal":
        return {"kind": kind, "n": 2 * _log_int(rng, 48, 256), "nsrc": _log_int(rng, 32, 128),
                "nvis": _log_int(rng, 3e4, 2e6), "term": rng.choice(["visibilities", "bcb"])}
    if kind == "solve":
        return {"kind": kind, "n": 2 * _log_int(rng, 64, 224), "nsrc": _log_int(rng, 48, 112),
                "nvis": _log_int(rng, 1e5, 1.5e6), "strength": 1e4, "tol": 1e-8}
    if kind == "deflect":
        return {"kind": kind, "points": _log_int(rng, 128 * 128, 60 * 512 * 512),
                "order": rng.choice([0, 3, 4])}
    if kind == "sweep":
        return {"kind": kind, "samples": rng.randint(3, 19), "layout": rng.randint(0, 9999)}
    if kind == "precondition":
        return {"kind": kind, "h": 8 * rng.randint(8, 20), "wd": 8 * rng.randint(8, 20)}
    return {"kind": kind, "h": 8 * rng.randint(8, 16), "wd": 8 * rng.randint(8, 16),
            "batch": rng.randint(1, 31)}


# ------------------------------------------------------------------------------------------------
# Inputs from the seed
# ------------------------------------------------------------------------------------------------
def _image_space(nx, ny, pix, off=0.0):
    hx, hy = 0.5 * nx * pix, 0.5 * ny * pix
    return ImageSpace((nx, ny), [(off - hx, off + hx), (0.5 * off - hy, 0.5 * off + hy)])


def _uv(rng, nvis, four, frac, w, blobs=0.0):
    """uv points with density ~ 1/|uv|, as a measurement set has them in wavelengths."""
    if blobs:
        return synthetic.synth_uv_blobs(rng, nvis, four, frac, w, blob_frac=blobs)
    return synthetic.synth_uv(rng, nvis, four, frac, w)


def _lens_parameters(rng, order=0):
    """(b, q, gamma, th, x, y), (ss, sa), multipole coefficients from the sweep's priors."""
    pemd = (rng.uniform(0.8, 1.6), rng.uniform(0.5, 0.95), rng.uniform(1.8, 2.3),
            rng.uniform(0.0, 180.0), rng.uniform(-0.05, 0.05), rng.uniform(-0.05, 0.05))
    shear = (rng.uniform(0.0, 0.1), rng.uniform(0.0, 180.0))
    coeff = rng.normal(0.0, 0.01, (max(0, order - 2), 2))
    return pemd, shear, coeff


def _lens_model(pemd, shear, coeff):
    b, q, gamma, th, x, y = pemd
    qh = 0.5 * (gamma - 1.0)
    parts = [PowerLawEllipsoid(z=0.5, b=b, th=th, f=q, x=x, y=y, rc=0.0, qh=qh),
             ExternalPotential(z=0.5, x=x, y=y, ss=shear[0], sa=shear[1])]
    if len(coeff):
        parts.append(InternalMultipoles(z=0.5, x=x, y=y, qh=qh, order=2 + len(coeff),
                                        coefficients=coeff))
    return GlobalLensModel(parts)


def _source_space(nsrc):
    return ImageSpace((nsrc, nsrc), [(-0.64, 0.64), (-0.64, 0.64)])


def _nufft_inputs(case, seed):
    rng = np.random.default_rng(seed)
    ims = _image_space(case["nx"], case["ny"], case["pix"], case["off"])
    four = synthetic.padded_fourier_space(ims, 2)
    uvw = _uv(rng, case["nvis"], four, 0.45, case["w"])
    return ims, four, uvw, rng.normal(size=(case["nx"], case["ny"]))


def _plan_inputs(case, seed):
    rng = np.random.default_rng(seed)
    ims = _image_space(case["n"], case["n"], 0.02)
    four = synthetic.padded_fourier_space(ims, 2)
    rows = case["nvis"] if case["kind"] == "grid" else case["nrows"]
    uvw = _uv(rng, rows, four, 0.48 if case["kind"] == "grid" else 0.45, case["w"],
              case.get("blobs", 0.0))
    channels = np.linspace(1.0, 0.9, case["nch"]) if case.get("nch", 1) > 1 else np.ones(1)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    grid = torch.randn((four.nu, four.nv // 2 + 1), dtype=torch.complex64, device="cuda",
                       generator=gen)
    vis = torch.randn(rows * channels.size, dtype=torch.complex128, device="cuda",
                      generator=gen)
    return four, uvw, channels, grid, vis


def _beta_2w(w):
    return 2.34 * 2 * w


def _inversion_inputs(case, seed):
    """The inversion's inputs but the data: image and source spaces, uv, sigma, lens
    parameters, and a vector on the source grid. The lens of the workload inversion, its
    parameters moved by the seed."""
    rng = np.random.default_rng(seed)
    ims = _image_space(case["n"], case["n"], 5.12 / case["n"])
    four = synthetic.padded_fourier_space(ims, 2)
    uvw = _uv(rng, case["nvis"], four, 0.45, 4)
    c = 0.0025 + 1e-4 * rng.uniform(-1, 1, 2)
    pemd = (1.2 + 0.02 * rng.uniform(-1, 1), 0.7, 2.0, 0.0, c[0], c[1])
    lens = (pemd, (0.05, 20.0), np.zeros((0, 2)))
    sigma = rng.uniform(0.8, 1.25, case["nvis"])
    return rng, ims, _source_space(case["nsrc"]), uvw, sigma, lens


def _inversion(case, seed):
    rng, ims, srcs, uvw, sigma, lens = _inversion_inputs(case, seed)
    vs = VisibilitySpace(channels=[1.0], uvcoords=uvw)
    nufft = NUFFTOperator(vs, ims)
    glm = _lens_model(*lens)
    xs = (srcs.xmin + srcs.dx * np.arange(srcs.nx))[:, None]
    ys = (srcs.ymin + srcs.dy * np.arange(srcs.ny))[None, :]
    src = (np.exp(-((xs - 0.05) ** 2 + (ys - 0.02) ** 2) / (2 * 0.06 ** 2))
           + 0.5 * np.exp(-((xs + 0.1) ** 2 + (ys + 0.08) ** 2) / (2 * 0.04 ** 2)))
    model = nufft * (BilinearLensOperator(ims, srcs, glm, Z_SRC) * src)
    data = model.reshape(-1) + sigma * synthetic.complex_normal(rng, case["nvis"])
    return SourceInversion(vs, data, sigma, ims, srcs, glm, Z_SRC,
                           case.get("strength", PRIOR), nufft=nufft,
                           data_term=case.get("term", "visibilities"))


def _source_vector(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    return torch.randn(case["nsrc"] ** 2, dtype=torch.float32, device="cuda", generator=g)


def _points(case, seed):
    """Image-plane positions over +-2.56 arcsec."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.rand((case["points"], 2), dtype=torch.float32, device="cuda", generator=g)
            - 0.5) * 5.12


def _sweep_samples(case, seed):
    """Samples of the sweep workload: image sizes and visibility counts by the case, lens
    parameters and uv draws by the seed."""
    samples = draw_samples(np.random.default_rng(seed), case["samples"])
    for s, size in zip(samples, draw_samples(np.random.default_rng(case["layout"]),
                                             case["samples"])):
        s.n, s.nvis, s.tol = size.n, size.nvis, size.tol
    return samples


def _sweep_data(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed + 2)
    return [torch.randn(s.nvis, dtype=torch.complex64, device="cuda", generator=g)
            for s in _sweep_samples(case, seed)]


LAYERS = [(2, 32, 3), (32, 64, 3), (64, 128, 3), (128, 128, 3), (128, 64, 1), (64, 32, 3),
          (32, 32, 3), (32, 1, 1)]


def _net_parameters(seed):
    rng = np.random.default_rng(seed)
    parts = []
    for ci, co, k in LAYERS:
        parts.append(rng.normal(0.0, math.sqrt(2.0 / (ci * k * k)), co * k * k * ci))
        parts.append(rng.normal(0.0, 0.05, co))
    return np.concatenate(parts).astype(np.float32)


def _net_inputs(case, seed):
    """A smooth scaled residual, the log-diagonal feature and a target, batched."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    shape = (case.get("batch", 1), case["h"], case["wd"])
    x, f, t = (torch.randn(shape, dtype=torch.float32, device="cuda", generator=g)
               for _ in range(3))
    return x, f - f.mean(), t


def _residual(case, seed):
    """A residual and an inverse Jacobi diagonal of uneven scale."""
    x, f, _ = _net_inputs(case, seed)
    dinv = torch.exp(0.7 * f[0]) * 1e-4
    return x[0] * 30.0, dinv


# ------------------------------------------------------------------------------------------------
# prepare and run
# ------------------------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "nufft":
        ims, four, uvw, image = _nufft_inputs(case, seed)
        op = NUFFTOperator(VisibilitySpace(channels=[1.0], uvcoords=uvw), ims,
                           kernel_support=case["w"], kb_beta=case["beta"] or None)
        return kind, op, torch.as_tensor(image, dtype=getattr(torch, case["dtype"])).cuda()
    if kind in ("grid", "rows"):
        four, uvw, channels, grid, vis = _plan_inputs(case, seed)
        plan = GriddingPlan(torch.as_tensor(uvw).cuda(), channels, four.nu, four.nv, four.du,
                            four.dv, four.gcx, four.gcy, case["w"], _beta_2w(case["w"]))
        return kind, plan, grid, vis
    if kind == "normal":
        return kind, _inversion(case, seed), _source_vector(case, seed)
    if kind == "solve":
        return kind, _inversion(case, seed), case["tol"]
    if kind == "deflect":
        lens = _lens_parameters(np.random.default_rng(seed), case["order"])
        return kind, _lens_model(*lens), _points(case, seed)
    if kind == "sweep":
        sweep = BatchedSweep(_sweep_samples(case, seed), seed=seed + 1)
        for plan, v, user in zip(sweep.plans, sweep.vis_in, _sweep_data(case, seed)):
            v.copy_(plan.to_plan(user))
        return kind, sweep
    net = UNet(case["h"], case["wd"], max_batch=case.get("batch", 1),
               params=_net_parameters(seed))
    if kind == "precondition":
        r, dinv = _residual(case, seed)
        return kind, net, r, dinv, features(dinv)
    return (kind, net) + _net_inputs(case, seed)


def run(state):
    kind = state[0]
    if kind == "nufft":
        _, op, image = state
        return op.T * (op * image)
    if kind == "grid":
        _, plan, grid, _ = state
        return plan.grid(plan.degrid(grid))
    if kind == "rows":
        _, plan, grid, vis = state
        model = plan.from_plan(plan.degrid(grid), dtype=torch.complex64)
        return {"model": model, "dirty": plan.grid(plan.to_plan(vis))}
    if kind == "normal":
        _, inv, s = state
        return inv.apply(s)
    if kind == "solve":
        _, inv, tol = state
        x, _ = inv.solve_flexible(tol=tol, inner_tol=1e-3, window=8)
        return x.float()  # the source image as it is kept
    if kind == "deflect":
        _, glm, points = state
        return glm.deflect(points, Z_SRC)
    if kind == "sweep":
        _, sweep = state
        sweep.run()
        torch.cuda.current_stream().wait_stream(sweep.stream)
        model = [p.from_plan(v, dtype=torch.complex64)
                 for p, v in zip(sweep.plans, sweep.vis_out)]
        return {"model": model, "grid": sweep.grid_out, "beta": sweep.beta_out}
    if kind == "precondition":
        _, net, r, dinv, feat = state
        return net.precondition(r, dinv, feat)
    _, net, x, f, t = state
    grad, loss = net.gradients(x, f, t)
    return {"grad": grad, "loss": loss}


# ------------------------------------------------------------------------------------------------
# What a pass cannot do without
# ------------------------------------------------------------------------------------------------
def _grid_work(nvis, w, ncells, value):
    """Degrid + grid: coordinates once per direction, visibilities and grid once each way."""
    return 2 * (nvis * (8 + value) + ncells * value), 2 * nvis * (4 * (2 * w) ** 2 + 80 * w)


def _fft_flops(n):
    return 2.5 * n * math.log2(n)


def work(case):
    kind = case["kind"]
    if kind == "nufft":
        w, value = case["w"], 8 if case["dtype"] == "float32" else 16
        npix, ngrid = case["nx"] * case["ny"], 4 * case["nx"] * case["ny"]
        b, f = _grid_work(case["nvis"], w, 0, value)
        return {"bytes": b + npix * value, "flops": f + 2 * _fft_flops(ngrid)}
    if kind == "grid":
        b, f = _grid_work(case["nvis"], case["w"], 2 * case["n"] ** 2, 8)
        return {"bytes": b, "flops": f}
    if kind == "rows":
        nvis = case["nrows"] * case["nch"]
        b, f = _grid_work(nvis, case["w"], 2 * case["n"] ** 2, 8)
        return {"bytes": b + 8 * nvis, "flops": f}
    if kind in ("normal", "solve"):
        n, nsrc = case["n"] ** 2, case["nsrc"] ** 2
        if case.get("term") == "bcb":
            b, f = 8 * 2 * n + 16 * n, 2 * _fft_flops(4 * n)
        else:
            b, f = _grid_work(case["nvis"], 4, 0, 8)
            b, f = b + 4 * case["nvis"], f + 2 * _fft_flops(4 * n)
        b, f = b + 2 * 32 * n + 8 * nsrc, f + 16 * n + 20 * nsrc
        if kind == "solve":  # about 100 matvecs
            b, f = 100 * b, 100 * f
        return {"bytes": b, "flops": f}
    if kind == "deflect":
        return {"bytes": 16 * case["points"],
                "flops": (150 + 40 * max(0, case["order"] - 2)) * case["points"]}
    if kind == "sweep":
        nvis, npix = 630000 * case["samples"], 123000 * case["samples"]
        b, f = _grid_work(nvis, 3.3, 2 * npix, 8)
        return {"bytes": b + 16 * nvis + 8 * npix, "flops": f + 150 * npix}
    npix = case["h"] * case["wd"]
    scale = {1: 1, 2: 4, 3: 16, 4: 64}
    level = [1, 2, 3, 4, 3, 2, 1, 1]
    flops = sum(2 * npix / scale[lv] * ci * co * k * k for (ci, co, k), lv in zip(LAYERS, level))
    params = sum(co * k * k * ci + co for ci, co, k in LAYERS)
    if kind == "precondition":
        return {"bytes": 2 * params + 16 * npix, "flops": flops}
    return {"bytes": case["batch"] * npix * 12 + 6 * params, "flops": 3 * case["batch"] * flops}


# ------------------------------------------------------------------------------------------------
# The same in 64 bits, from the definitions
# ------------------------------------------------------------------------------------------------
class _Gridder:
    """Kaiser-Bessel interpolation between visibilities and the half-plane grid, by its sum over
    taps: weight I0(beta sqrt(1 - (a/w)^2)) / (2w) per axis, taps round(g) - w ... round(g) + w,
    checkerboard sign, Hermitian fold."""

    def __init__(self, uvw, channels, four, w, beta):
        uvw = torch.as_tensor(uvw).cuda()
        ch = torch.as_tensor(np.asarray(channels, dtype=np.float64)).cuda()
        u = (ch[:, None] * uvw[None, :, 0]).reshape(-1)
        v = -(ch[:, None] * uvw[None, :, 1]).reshape(-1)
        phase = TWO_PI * (u * four.gcx + v * four.gcy)
        self.phase = torch.polar(torch.ones_like(phase), phase)
        self.nu, self.nv, self.half = four.nu, four.nv, four.nv // 2 + 1
        self.w, self.beta = w, beta
        self.gu, self.gv = u / four.du, v / four.dv
        self.cu, self.cv = torch.round(self.gu).long(), torch.round(self.gv).long()

    def _taps(self, g, c):
        a = g[None, :] - (c[None, :] + torch.arange(-self.w, self.w + 1, device="cuda")[:, None])
        k = torch.special.i0(self.beta * torch.sqrt((1 - (a / self.w) ** 2).clamp(min=0)))
        return torch.where(a.abs() <= self.w, k / (2 * self.w), torch.zeros_like(k))

    def _each(self):
        ku, kv = self._taps(self.gu, self.cu), self._taps(self.gv, self.cv)
        for i in range(2 * self.w + 1):
            tu = self.cu + i - self.w
            row = torch.remainder(tu, self.nu) * self.nv
            for j in range(2 * self.w + 1):
                tv = self.cv + j - self.w
                yield row + torch.remainder(tv, self.nv), \
                    ku[i] * kv[j] * (1 - 2 * torch.remainder(tu + tv, 2))

    def _mirror(self, x):
        """x[(nu - i) % nu, (nv - j) % nv]"""
        return torch.roll(torch.flip(x, (0, 1)), (1, 1), (0, 1))

    def forward(self, grid):
        full = torch.zeros((self.nu, self.nv), dtype=torch.complex128, device="cuda")
        full[:, :self.half] = grid
        full[:, self.half:] = self._mirror(full).conj()[:, self.half:]
        full = full.reshape(-1)
        out = torch.zeros_like(self.phase)
        for at, k in self._each():
            out += k * full[at]
        return out * self.phase.conj()

    def adjoint(self, vis):
        acc = torch.zeros((self.nu * self.nv, 2), dtype=torch.float64, device="cuda")
        val = torch.view_as_real(0.5 * vis * self.phase)
        for at, k in self._each():
            acc.index_add_(0, at, k[:, None] * val)
        acc = torch.view_as_complex(acc).reshape(self.nu, self.nv)
        out = acc[:, :self.half].clone()
        out[:, 0] *= 2
        top = self.nv - self.half  # columns 1 ... top have a partner beyond the half plane
        out[:, 1:top + 1] += self._mirror(acc).conj()[:, 1:top + 1]
        return out


class _Nufft:
    """Apodisation, zero padding, real FFT and gridding of an image space."""

    def __init__(self, uvw, ims, w, beta=None):
        self.pad = ((ims.nx + 1) // 2, (ims.ny + 1) // 2)
        self.shape = (ims.nx + 2 * self.pad[0], ims.ny + 2 * self.pad[1])
        beta = beta or math.pi * math.sqrt((2.0 * w / 2) ** 2 * 1.5 ** 2 - 0.8)
        four = synthetic.padded_fourier_space(ims, 2)
        self.ims, self.gridder = ims, _Gridder(uvw, [1.0], four, w, beta)

        def correction(n, m):
            c = (torch.arange(n, dtype=torch.float64, device="cuda") - 0.5 * n) / m
            s = torch.sqrt(beta ** 2 - (2 * math.pi * w * c) ** 2)
            return s / torch.sinh(s)
        self.apod = torch.outer(correction(ims.nx, self.shape[0]),
                                correction(ims.ny, self.shape[1]))

    def forward(self, image):
        z = torch.zeros(self.shape, dtype=torch.float64, device="cuda")
        px, py = self.pad
        z[px:px + self.ims.nx, py:py + self.ims.ny] = self.apod * image
        return self.gridder.forward(torch.fft.rfft2(z))

    def adjoint(self, vis):
        y = torch.fft.irfft2(self.gridder.adjoint(vis), s=self.shape, norm="forward")
        px, py = self.pad
        return self.apod * y[px:px + self.ims.nx, py:py + self.ims.ny]


def _deflected(points, pemd, shear, coeff):
    """Source-plane positions by the 20-term series of the power-law ellipsoid, external shear
    and internal multipoles."""
    p = points.double()
    b, q, gamma, th, x0, y0 = pemd
    t = gamma - 1.0
    d = torch.view_as_complex((p - torch.tensor([x0, y0], dtype=torch.float64,
                                                device=p.device)).contiguous())
    bn = (0.5 * b * q ** (t - 0.5) * (3.0 - t) / (2.0 - t)) ** (1.0 / t)
    ang = (th + 90) * math.pi / 180
    rot = complex(math.cos(ang), -math.sin(ang))
    z = d * rot
    rs = torch.sqrt(q * q * z.real ** 2 + z.imag ** 2)
    u = 0.5 * (1.0 - torch.sqrt(1.0 - (1 - q * q) / (q * q) * rs ** 2 / (z * z)))
    f, un, an = torch.zeros_like(z), torch.ones_like(z), 1.0
    for n in range(20):
        f = f + an * un
        un = un * u
        an *= (2 * n + 4 - 2 * t) / (2 * n + 4 - t)
    alpha = (bn * bn / (q * z) * (bn / rs) ** (t - 2) * f * rot).conj()
    ss, sa = shear
    s, c = math.sin((sa + 90) * math.pi / 180), math.cos((sa + 90) * math.pi / 180)
    c2, s2 = s * s - c * c, -2 * s * c
    alpha = alpha + ss * torch.complex(c2 * d.real + s2 * d.imag, s2 * d.real - c2 * d.imag)
    r, e = d.abs(), d / d.abs()
    for i, (am, bm) in enumerate(coeff):
        m = i + 3
        em = e ** m
        norm = 2.0 / (m * m - (t - 2) ** 2) * r ** (1.0 - t)
        dr = -norm * (2.0 - t) * (bm * em.imag + am * em.real)
        dt = norm * m * (-bm * em.real + am * em.imag)
        alpha = alpha + e * torch.complex(dr, dt)
    return p - torch.view_as_real(alpha)


def _bilinear(points, srcs):
    """(source indices, weights) (npix, 4) of the bilinear lens operator; weight 0 outside."""
    fx, fy = (points[:, 0] - srcs.xmin) / srcs.dx, (points[:, 1] - srcs.ymin) / srcs.dy
    j, k = torch.floor(fx), torch.floor(fy)
    ok = (j >= 0) & (j <= srcs.nx - 2) & (k >= 0) & (k <= srcs.ny - 2)
    tx, ty = fx - j, fy - k
    j, k = (torch.where(ok, a, torch.zeros_like(a)).long() for a in (j, k))
    at = torch.stack([j * srcs.ny + k, (j + 1) * srcs.ny + k, j * srcs.ny + k + 1,
                      (j + 1) * srcs.ny + k + 1], 1)
    wt = torch.stack([(1 - tx) * (1 - ty), tx * (1 - ty), (1 - tx) * ty, tx * ty], 1)
    return at, torch.where(ok[:, None], wt, torch.zeros_like(wt))


def _gradient_prior(s, srcs, strength):
    s = s.reshape(srcs.nx, srcs.ny)
    out = torch.zeros_like(s)
    for dim, h in ((0, srcs.dx), (1, srcs.dy)):
        g = torch.diff(s, dim=dim) / (h * h)
        n = s.shape[dim] - 1
        out.narrow(dim, 0, n).sub_(g)
        out.narrow(dim, 1, n).add_(g)
    return strength * out.reshape(-1)


def _exact_normal(case, seed):
    _, ims, srcs, uvw, sigma, lens = _inversion_inputs(case, seed)
    s = _source_vector(case, seed).double()
    points = torch.as_tensor(ims.points.reshape(-1, 2)).cuda()
    at, wt = _bilinear(_deflected(points, *lens), srcs)
    image = (wt * s[at]).sum(1).reshape(ims.nx, ims.ny)
    weights = torch.as_tensor(sigma).cuda() ** -2
    if case["term"] == "bcb":
        rx, ry = ims.dx * ims.nx, ims.dy * ims.ny
        beam = _Nufft(uvw, ImageSpace((2 * ims.nx, 2 * ims.ny), [(-rx, rx), (-ry, ry)]),
                      4).adjoint(weights.to(torch.complex128))
        beam = torch.roll(beam, (ims.nx, ims.ny), (0, 1))
        z = torch.zeros_like(beam)
        inner = (slice(ims.nx // 2, ims.nx // 2 + ims.nx),
                 slice(ims.ny // 2, ims.ny // 2 + ims.ny))
        z[inner] = image
        y = torch.fft.irfft2(torch.fft.rfft2(beam) * torch.fft.rfft2(z), s=z.shape)[inner]
    else:
        nufft = _Nufft(uvw, ims, 4)
        y = nufft.adjoint(weights * nufft.forward(image))
    out = torch.zeros_like(s)
    out.index_add_(0, at.reshape(-1), (wt * y.reshape(-1, 1)).reshape(-1))
    return out + _gradient_prior(s, srcs, PRIOR)


def _net(params, x, f):
    """The U-Net in 64 bits: three pooled levels, nearest-neighbour upsampling, additive
    skips. Returns the output (B, H, W)."""
    Fn = torch.nn.functional
    layers, o = [], 0
    for ci, co, k in LAYERS:
        n = co * k * k * ci
        layers.append((params[o:o + n].reshape(co, k, k, ci).permute(0, 3, 1, 2),
                       params[o + n:o + n + co]))
        o += n + co

    def conv(i, a):
        w, b = layers[i]
        co, ci, k, _ = w.shape
        cols = Fn.unfold(a, k, padding=k // 2)  # a plain contraction in FP64
        y = torch.einsum("ok,bkp->bop", w.reshape(co, -1), cols) + b[:, None]
        y = y.reshape(a.shape[0], co, *a.shape[2:])
        return y if i == 7 else torch.relu(y)

    def up(a):
        return a.repeat_interleave(2, 2).repeat_interleave(2, 3)

    e1 = conv(0, torch.stack([x, f], 1))
    e2 = conv(1, Fn.avg_pool2d(e1, 2))
    e3 = conv(2, Fn.avg_pool2d(e2, 2))
    c3 = conv(4, up(conv(3, Fn.avg_pool2d(e3, 2))) + e3)
    c2 = conv(5, up(c3) + e2)
    return conv(7, conv(6, up(c2) + e1))[:, 0]


def exact(case, seed):
    kind = case["kind"]
    if kind == "nufft":
        ims, _, uvw, image = _nufft_inputs(case, seed)
        image = torch.as_tensor(image, dtype=getattr(torch, case["dtype"])).cuda().double()
        op = _Nufft(uvw, ims, case["w"], case["beta"])
        return op.adjoint(op.forward(image))
    if kind in ("grid", "rows"):
        four, uvw, channels, grid, vis = _plan_inputs(case, seed)
        g = _Gridder(uvw, channels, four, case["w"], _beta_2w(case["w"]))
        model = g.forward(grid.to(torch.complex128))
        if kind == "grid":
            return g.adjoint(model)
        return {"model": model, "dirty": g.adjoint(vis)}
    if kind == "normal":
        return _exact_normal(case, seed)
    if kind == "solve":
        return None  # hundreds of operator applications in 64 bits
    if kind == "deflect":
        lens = _lens_parameters(np.random.default_rng(seed), case["order"])
        points = _points(case, seed)
        return torch.cat([_deflected(p, *lens) for p in points.split(1 << 22)])
    if kind == "sweep":
        samples, out = _sweep_samples(case, seed), {"model": [], "grid": [], "beta": []}
        gen = torch.Generator(device="cuda").manual_seed(seed + 1)
        for s, user in zip(samples, _sweep_data(case, seed)):
            ims = _image_space(s.n, s.n, s.pix)
            four = synthetic.padded_fourier_space(ims, 2)
            w = 3 if s.tol >= 1.2e-5 else 4  # kernel width by the sample's accuracy target
            uvw = synthetic.synth_uv(np.random.default_rng(s.seed), s.nvis, four, 0.45, w)
            grid = torch.randn((four.nu, four.nv // 2 + 1), dtype=torch.complex64,
                               device="cuda", generator=gen)
            torch.randn(s.nvis, dtype=torch.complex64, device="cuda", generator=gen)
            g = _Gridder(uvw, [1.0], four, w, _beta_2w(w))
            out["model"].append(g.forward(grid.to(torch.complex128)))
            out["grid"].append(g.adjoint(user.to(torch.complex128)))
            c = -0.5 * s.n * s.pix + 0.5 * s.pix + s.pix * torch.arange(
                s.n, dtype=torch.float64, device="cuda")
            pemd, shear = s.lenses
            out["beta"].append(_deflected(
                torch.cartesian_prod(c, c),
                (pemd.b, pemd.f, 2 * pemd.qh + 1, pemd.th, pemd.x, pemd.y),
                (shear.ss, shear.sa), ()))
        return out
    params = torch.as_tensor(_net_parameters(seed)).cuda().double()
    if kind == "precondition":
        r, dinv = (a.double() for a in _residual(case, seed))
        u = r * dinv
        s = u.square().mean().sqrt()
        f = torch.log(dinv)
        return s * _net(params, (u / s)[None], (f - f.mean())[None])[0]
    x, f, t = (a.double() for a in _net_inputs(case, seed))
    params.requires_grad_(True)
    loss, parts = 0.0, max(1, case["batch"] // 4)
    for a, b, c in zip(x.chunk(parts), f.chunk(parts), t.chunk(parts)):
        part = (_net(params, a, b) - c).square().sum() / t.numel()
        part.backward()
        loss += float(part)
    return {"grad": params.grad, "loss": loss}
