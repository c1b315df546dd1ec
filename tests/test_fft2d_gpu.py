"""The padded real transforms of power-of-two planes (csrc/fft2d.cu) inside the NUFFT and the
dirty-beam convolution, against the FP64 oracle: every length the kernels have (128 to 2048) as
rows and as columns, images of half and of a quarter of the plane, and the first length beyond
them on the library transform.

Tolerances. FP64: the degree-11 fits of the weights are within 4.5e-13 of the profile's peak at
w = 4, about three times the rms weight: 1.4e-12 relative, and log2(2048 * 128) = 18 roundings of
2^-53 beside it. FP32: at most 18 stages and 72 taps of 2^-24 in the mean square:
sqrt(90) * 2^-24 = 5.7e-7."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,pad", [(64, 64, 2), (64, 128, 2), (256, 64, 2), (64, 512, 2),
                                       (1024, 64, 2), (64, 1024, 2), (512, 64, 2), (32, 64, 4),
                                       (128, 2048, 2)])
def test_nufft(native, nx, ny, pad):
    from lentils_gb300.operators import NUFFTOperator
    from lentils_gb300.spaces import ImageSpace, VisibilitySpace
    rng = np.random.default_rng(nx + ny)
    b = [(-0.5, 0.3), (-0.2, 0.9)]
    img = O.ImageGeom((nx, ny), b)
    padded, _, _ = O.padded_geom(img, pad)
    uvw = O.synth_uv(rng, 1500, O.FourierGeom(padded), 0.45, 4)
    ora = O.NufftOracle(O.VisGeom(uvw, [1.0]), img, pad, 4)
    op = NUFFTOperator(VisibilitySpace([1.0], uvw), ImageSpace((nx, ny), b), pad, 4)
    x = rng.normal(size=(nx, ny))
    v = rng.normal(size=1500) + 1j * rng.normal(size=1500)
    y, z = (op * x).reshape(-1), (op.T * v).reshape(nx, ny)
    ry, rz = ora.forward(x), ora.adjoint(v)
    assert O.rel_l2(y, ry) < 2e-7 and O.rel_l2(z, rz) < 2e-7  # FP32 phases (off-centre image)
    # without the phases: F^T F in plan order
    x64 = torch.as_tensor(x).cuda()
    rn = ora.adjoint(ry)
    assert O.rel_l2((op.T * (op * x64)).cpu().numpy(), rn) < 3e-12
    assert O.rel_l2((op.T * (op * x64.float())).cpu().numpy(), rn) < 1.2e-6


@pytest.mark.parametrize("nx,ny", [(64, 64), (64, 256), (512, 64), (64, 1024), (1024, 64)])
def test_convolution(native, nx, ny):
    from lentils_gb300.operators import BlurredCovarianceOperator
    from lentils_gb300.spaces import ImageSpace, VisibilitySpace
    rng = np.random.default_rng(nx + 3 * ny)
    b = [(-0.4, 0.4), (-0.6, 0.6)]
    img = O.ImageGeom((nx, ny), b)
    padded, _, _ = O.padded_geom(img, 2)
    uvw = O.synth_uv(rng, 2000, O.FourierGeom(padded), 0.3, 4)
    w = rng.uniform(0.5, 2.0, 2000)
    op = BlurredCovarianceOperator(VisibilitySpace([1.0], uvw), ImageSpace((nx, ny), b), w)
    x = rng.normal(size=(nx, ny))
    ref = O.bcb_apply(op.dirty_beam, img, x)
    assert O.rel_l2(op * x, ref) < 1e-14
    got = op * torch.as_tensor(x, dtype=torch.float32).cuda()
    assert O.rel_l2(got.cpu().numpy(), ref) < 5.7e-7


@pytest.mark.parametrize("real,cplx,tol", [(torch.float32, torch.complex64, 1.2e-6),
                                           (torch.float64, torch.complex128, 3e-12)])
def test_adjoint_leaves_its_grid_zero(native, real, cplx, tol):
    """The adjoint accumulates into a grid that its own column transform leaves zero: repeated, with
    forward calls between, and captured and replayed, each call gives the adjoint of its own input.
    Tolerances as above."""
    from lentils_gb300.operators import NUFFTOperator
    from lentils_gb300.spaces import ImageSpace, VisibilitySpace
    rng = np.random.default_rng(12)
    n, b = 64, [(-0.5, 0.3), (-0.2, 0.9)]
    img = O.ImageGeom((n, n), b)
    padded, _, _ = O.padded_geom(img, 2)
    uvw = O.synth_uv(rng, 1500, O.FourierGeom(padded), 0.45, 4)
    ora = O.NufftOracle(O.VisGeom(uvw, [1.0]), img, 2, 4)
    op = NUFFTOperator(VisibilitySpace([1.0], uvw), ImageSpace((n, n), b), 2, 4)
    xs = [rng.normal(size=(n, n)) for _ in range(2)]
    ref = [ora.adjoint(ora.forward(x)).reshape(n, n) for x in xs]
    ys = [(op * torch.as_tensor(x).cuda()).to(cplx) for x in xs]

    def check(got, i):
        assert O.rel_l2(got.cpu().numpy(), ref[i]) < tol
    for i in (0, 1, 1, 0):
        check(op.T * ys[i], i)
        op * torch.as_tensor(xs[1 - i], dtype=real).cuda()
    static = ys[0].clone()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(s):
        op.T * static
        torch.cuda.synchronize()
        with torch.cuda.graph(g, stream=s):
            out = op.T * static
    torch.cuda.current_stream().wait_stream(s)
    for i in (0, 1, 0):
        static.copy_(ys[i])
        g.replay()
        check(out, i)
        check(op.T * ys[1 - i], 1 - i)
