"""The paired-FP32 form of the FP64 operators (csrc/gridding64.cu) against a plain FP64 sum with
the same fits of the weights (12 Chebyshev nodes per tap; 10 in the FP64 kernels of the other
plans), so that what is left is the pairs' own rounding.

Tolerance: a multiply-add of pairs is good to 2^-47 of the larger of its terms. A result is at
most (2w)^2 + 2w = 72 of them in a row (gridding: one per visibility of a run, and the sums of
runs), whose errors add at worst linearly: 72 * 2^-47 = 5.1e-13; the weights, on a grid of 2^-23
of a bias of a few times their largest value, are good to about 2^-43 = 1.1e-13 of their
peak."""
import ctypes

import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu
TOL = 7e-13


def weights(f, w, beta, n):
    """(2w, f.size): the interpolants at n Chebyshev nodes of I0(beta sqrt(1 - (a/w)^2)) / (2w),
    tap i at argument a = f + w - 1 - i."""
    nodes = 0.5 * (np.cos(np.pi * (np.arange(n) + 0.5) / n) + 1)
    out = np.empty((2 * w, f.size))
    for i in range(w):
        a = (nodes + w - 1 - i) / w
        c = np.polynomial.chebyshev.chebfit(2 * nodes - 1, np.i0(beta * np.sqrt(1 - a * a)),
                                            n - 1)
        out[i] = np.polynomial.chebyshev.chebval(2 * f - 1, c) / (2 * w)
        out[2 * w - 1 - i] = np.polynomial.chebyshev.chebval(1 - 2 * f, c) / (2 * w)
    return out


class Direct:
    def __init__(self, uvw, four, w, beta, n=12):
        self.four, self.w = four, w
        self.axes = []
        for g, size in ((uvw[:, 0] / four.du, four.nu),
                        (-uvw[:, 1] / four.dv, four.nv)):
            # the cell of the coordinate rounded to 2^-24 cells, and the reference's tap set,
            # |g - i| <= w in FP64 (nufft.c:12): a coordinate within 2^-25 below a cell boundary
            # belongs to the cell above it, with the extra tap at argument +w
            b = np.floor(np.rint(g * 2.0 ** 24) / 2.0 ** 24)
            wt = np.concatenate([(g - (b - w) <= w)[None] / (2.0 * w), weights(g - b, w, beta, n)])
            wt[-1, ~(g - (b + w) >= -w)] = 0
            # taps b - w (extra), b - w + 1 + i
            idx = b[None].astype(int) - w + np.arange(2 * w + 1)[:, None]
            self.axes.append((idx, wt * (1 - 2 * (idx & 1)), size))

    def _cells(self):
        (iu, wu, nu), (iv, wv, nv) = self.axes
        for a in range(2 * self.w + 1):
            for b in range(2 * self.w + 1):
                yield iu[a] % nu, iv[b] % nv, wu[a] * wv[b]

    def degrid(self, grid):
        f = self.four
        full = np.zeros((f.nu, f.nv), complex)
        full[:, :f.half_nv] = grid
        mir = np.roll(np.flip(full, (0, 1)), (1, 1), (0, 1)).conj()
        full[:, f.half_nv:] = mir[:, f.half_nv:]
        out = 0
        for u, v, k in self._cells():
            out = out + k * full[u, v]
        return out

    def grid(self, vis):
        f = self.four
        acc = np.zeros((f.nu, f.nv), complex)
        for u, v, k in self._cells():
            np.add.at(acc, (u, v), 0.5 * k * vis)
        out = acc[:, :f.half_nv].copy()
        out[:, 0] *= 2
        mir = np.roll(np.flip(acc, (0, 1)), (1, 1), (0, 1)).conj()
        top = f.nv - f.half_nv
        out[:, 1:top + 1] += mir[:, 1:top + 1]
        return out


def setup(rng, nx, ny, w, nvis, tile, integer=0, chunk=0):
    from lentils_gb300.gridding import GriddingPlan
    img = O.ImageGeom((nx, ny), [(-1.0, 1.0), (-1.3, 1.3)])
    four = O.FourierGeom(img)
    beta = 2.34 * 2 * w
    uvw = O.synth_uv(rng, nvis, four, 0.45, w)
    uvw[:integer, 0] = np.round(uvw[:integer, 0] / four.du) * four.du
    uvw[:integer // 2, 1] = np.round(uvw[:integer // 2, 1] / four.dv) * four.dv
    plan = GriddingPlan(uvw, [1.0], four.nu, four.nv, four.du, four.dv, 0.0, 0.0, w, beta,
                        tile=tile, chunk=chunk)
    return four, Direct(uvw, four, w, beta, 12 if w <= 4 and tile <= 16 else 10), plan


def both(plan, four, grid, vis):
    from lentils_gb300 import _native as N
    sp = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    y = plan.degrid64(torch.as_tensor(grid).cuda())
    rows = torch.zeros(plan.nvis, dtype=torch.complex128, device="cuda")
    N.check(N.lib().lentils_vis_from_plan64(plan.handle, ptr(y), ptr(rows), 0, sp))
    user = torch.as_tensor(vis).cuda()
    vp = torch.empty_like(user)
    N.check(N.lib().lentils_vis_to_plan64(plan.handle, ptr(user), ptr(vp), sp))
    return rows.cpu().numpy(), plan.grid64(vp).cpu().numpy()


def cnormal(rng, *shape):
    return rng.normal(size=shape) + 1j * rng.normal(size=shape)


@pytest.mark.parametrize("w,tile,nx,ny,nvis,integer,chunk", [
    (1, 8, 40, 36, 1, 0, 0), (1, 16, 64, 48, 3000, 60, 0), (2, 8, 51, 47, 2500, 40, 256),
    (2, 16, 64, 64, 4097, 0, 4096), (3, 16, 75, 64, 3001, 30, 0), (3, 8, 64, 50, 129, 129, 0),
    (4, 16, 96, 80, 5003, 50, 1024), (4, 8, 81, 77, 2000, 0, 0), (4, 32, 96, 96, 2000, 10, 0),
    (5, 16, 96, 80, 2000, 10, 0)])
def test_against_direct_sum(native, w, tile, nx, ny, nvis, integer, chunk):
    """Widths and tiles with paired kernels and (the last two) on the FP64 kernels; grids of odd
    and even size; items of one and of many visibilities; coordinates on cell boundaries."""
    rng = np.random.default_rng(100 * w + tile)
    four, ref, plan = setup(rng, nx, ny, w, nvis, tile, integer, chunk)
    grid, vis = cnormal(rng, four.nu, four.half_nv), cnormal(rng, nvis)
    y, g = both(plan, four, grid, vis)
    assert O.rel_l2(y, ref.degrid(grid)) < TOL
    assert O.rel_l2(g, ref.grid(vis)) < TOL


@pytest.mark.parametrize("scale", [1e-290, 1e-40, 1e40, 1e280])
def test_range(native, scale):
    """Magnitudes beyond FP32's exponents, and values 1e8 apart side by side."""
    rng = np.random.default_rng(8)
    four, ref, plan = setup(rng, 64, 64, 4, 3000, 16)
    grid = scale * cnormal(rng, four.nu, four.half_nv) * 10 ** rng.uniform(-8, 0, (four.nu, 1))
    vis = scale * cnormal(rng, 3000) * 10 ** rng.uniform(-8, 0, 3000)
    y, g = both(plan, four, grid, vis)
    assert O.rel_l2(y / scale, ref.degrid(grid / scale)) < TOL
    assert O.rel_l2(g / scale, ref.grid(vis / scale)) < TOL


def test_not_finite(native):
    """An infinite and a NaN grid cell / visibility reach exactly the results they touch."""
    rng = np.random.default_rng(9)
    four, ref, plan = setup(rng, 64, 64, 3, 2000, 16)
    grid, vis = cnormal(rng, four.nu, four.half_nv), cnormal(rng, 2000)
    grid[5, 9], grid[40, 20] = np.inf, np.nan
    vis[7], vis[1200] = complex(np.nan, 0), complex(0, -np.inf)
    y, g = both(plan, four, grid, vis)
    with np.errstate(all="ignore"):
        ry, rg = ref.degrid(grid), ref.grid(vis)
    # numpy's complex products spread NaN over both parts, and its extra taps have weight 0:
    # compare by the cells with a nonzero weight
    touched = np.zeros(2000, bool)
    clean = grid.copy()
    clean[5, 9] = clean[40, 20] = 0
    for u, v, k in ref._cells():
        fold = v >= four.half_nv
        uu, vv = np.where(fold, (four.nu - u) % four.nu, u), np.where(fold, four.nv - v, v)
        touched |= (k != 0) & (((uu == 5) & (vv == 9)) | ((uu == 40) & (vv == 20)))
    assert touched.any() and np.array_equal(~np.isfinite(y), touched)
    assert O.rel_l2(y[~touched], ref.degrid(clean)[~touched]) < TOL
    bad = np.zeros((four.nu, four.half_nv), bool)
    for u, v, k in ref._cells():
        for i in (7, 1200):
            if k[i] != 0:
                fold = v[i] >= four.half_nv
                bad[(four.nu - u[i]) % four.nu if fold else u[i],
                    four.nv - v[i] if fold else v[i]] = True
    assert np.array_equal(~np.isfinite(g), bad)
    clean = vis.copy()
    clean[[7, 1200]] = 0
    assert O.rel_l2(g[~bad], ref.grid(clean)[~bad]) < TOL
