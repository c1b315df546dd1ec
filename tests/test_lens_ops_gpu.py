"""The lens operators' kernels (csrc/lens_ops.cu) where a thread or warp goes round more than once
and where the normal operator's transpose adds the gradient prior in the same pass: images beyond
one pixel per thread, source grids beyond one node per warp, a single row and a single column of
nodes, nodes of 0, 1, 32, 33 and 100 entries.

Tolerances. FP64: sums of at most 1e3 products, 1e3 * 2^-53 = 1e-13, with a margin of 10. FP32:
inputs, weights and products rounded to 2^-24 (three roundings), sums of at most 100 (seven levels
of a mean square each, sqrt(16) * 2^-24), and the beam's convolution 5.7e-7 beside them: 1e-6."""
import ctypes

import numpy as np
import pytest
import scipy.sparse as sps
import torch

import oracle as O

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("nsx,nsy", [(1, 77), (77, 1), (33, 31), (211, 200)])
def test_transpose_with_prior(native, nsx, nsy):
    from lentils_gb300 import _native as N
    rng = np.random.default_rng(nsx)
    L, sp = N.lib(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    n, nsrc, lam = 32, nsx * nsy, 0.03
    beam = rng.normal(size=(2 * n, 2 * n))
    lens = np.zeros(nsrc, int)  # entries of each node
    lens[rng.permutation(nsrc)[:70]] = np.tile([1, 3, 32, 33, 100, 31, 7], 10)
    lens[nsrc - 1] = 33
    cols = np.repeat(np.arange(nsrc), lens)
    rows = np.concatenate([rng.permutation(n * n)[:k] for k in lens if k])
    M = sps.csr_matrix((rng.normal(size=cols.size), (rows, cols)), shape=(n * n, nsrc))
    assert M.nnz == cols.size
    dev = [torch.as_tensor(a).cuda() for a in (M.indptr.astype(np.int32),
                                               M.indices.astype(np.int32), M.data, beam)]
    lo, bo, no = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_void_p()
    N.check(L.lentils_lensop_create_csr(ctypes.byref(lo), *map(_p, dev[:3]), n * n, nsrc, M.nnz, sp))
    N.check(L.lentils_bcb_create(ctypes.byref(bo), _p(dev[3]), n, n, sp))
    N.check(L.lentils_normal_op_create_bcb(ctypes.byref(no), lo, bo, n * n, nsx, nsy, 0.5, 0.25,
                                           lam, sp))
    try:
        s = rng.normal(size=nsrc)
        img = torch.as_tensor(M @ s).cuda()
        conv = torch.empty_like(img)
        N.check(L.lentils_bcb_apply64(bo, _p(img), _p(conv), sp))
        data = M.T @ conv.cpu().numpy()
        R = O.regulariser(O.ImageGeom((nsx, nsy), [(0, 0.5 * nsx), (0, 0.25 * nsy)]), 1.0)
        ref = data + lam * (R @ s)
        for dtype, fn, tol in ((torch.float64, L.lentils_normal_op_apply64, 1e-12),
                               (torch.float32, L.lentils_normal_op_apply, 1e-6)):
            x = torch.as_tensor(s, dtype=dtype).cuda()
            y = torch.full_like(x, float("nan"))
            N.check(fn(no, _p(x), _p(y), sp))
            got = y.double().cpu().numpy()
            assert O.rel_l2(got, ref) < tol
            empty = lens == 0
            assert O.rel_l2(got[empty], lam * (R @ s)[empty]) < tol or not empty.any()
    finally:
        torch.cuda.synchronize()
        L.lentils_normal_op_destroy(no)
        L.lentils_bcb_destroy(bo)
        L.lentils_lensop_destroy(lo)


def test_more_pixels_than_threads(native):
    from lentils_gb300 import _native as N
    rng = np.random.default_rng(4)
    L, sp = N.lib(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    nimg, src = 1_300_001, O.ImageGeom((60, 50), [(-1.0, 2.0), (-2.0, 3.0)])
    pts = rng.uniform(-2.5, 3.5, size=(nimg, 2))  # some outside the source grid
    mask = rng.random(nimg) < 0.9
    M = O.bilinear_lens_matrix(pts, mask, src)
    d_pts, d_mask = torch.as_tensor(pts).cuda(), torch.as_tensor(mask.astype(np.uint8)).cuda()
    lo = ctypes.c_void_p()
    N.check(L.lentils_lensop_create(ctypes.byref(lo), _p(d_pts), _p(d_mask), nimg, src.nx, src.ny,
                                    src.xmin, src.ymin, src.dx, src.dy, sp))
    try:
        s, r = rng.normal(size=src.nx * src.ny), rng.normal(size=nimg)
        for dtype, sfx, tol in ((torch.float64, "64", 1e-12), (torch.float32, "", 1e-6)):
            for x, ref, name in ((s, M @ s, "apply"), (r, M.T @ r, "apply_t")):
                d = torch.as_tensor(x, dtype=dtype).cuda()
                y = torch.full((ref.size,), float("nan"), dtype=dtype, device="cuda")
                N.check(getattr(L, f"lentils_lensop_{name}{sfx}")(lo, _p(d), _p(y), sp))
                assert O.rel_l2(y.double().cpu().numpy(), ref) < tol
    finally:
        torch.cuda.synchronize()
        L.lentils_lensop_destroy(lo)
