"""FP64 operators called in a row take no longer per call than one call by itself: a kernel that starts
while the one before it still runs must not have its CTAs packed onto the few SMs that are free."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu


def per_call(f, n):
    """Median time (us) of n calls in a row, divided by n; the host is ahead of the device."""
    for _ in range(3):
        f()
    times = []
    for _ in range(15):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        torch.cuda.synchronize()
        torch.cuda._sleep(2_000_000)
        a.record()
        for _ in range(n):
            f()
        b.record()
        b.synchronize()
        times.append(1e3 * a.elapsed_time(b) / n)
    return float(np.median(times))


@pytest.mark.parametrize("adjoint", [False, True])
@pytest.mark.parametrize("nx,ny,w", [(256, 256, 3), (64, 1024, 4)])
def test_calls_in_a_row(native, nx, ny, w, adjoint):
    from lentils_gb300.operators import NUFFTOperator
    from lentils_gb300.spaces import ImageSpace, VisibilitySpace
    rng = np.random.default_rng(nx)
    bounds = [(-0.01 * nx, 0.01 * nx), (-0.01 * ny, 0.01 * ny)]
    padded, _, _ = O.padded_geom(O.ImageGeom((nx, ny), bounds), 2)
    uvw = O.synth_uv(rng, 60000, O.FourierGeom(padded), 0.45, w)
    op = NUFFTOperator(VisibilitySpace([1.0], uvw), ImageSpace((nx, ny), bounds),
                       kernel_support=w)
    x = torch.randn((nx, ny), dtype=torch.float64, device="cuda")
    v = op * x
    f = (lambda: op.T * v) if adjoint else (lambda: op * x)
    one, many = per_call(f, 1), per_call(f, 20)
    assert many < 1.15 * one, (one, many)
