"""Operators whose constants are uploaded at their creation: the uploads are ordered before the
operator's kernels on every stream."""
import glob
import os
import re

import numpy as np
import pytest
import torch

import oracle as O

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lentils_gb300",
                    "csrc")


def test_no_upload_on_the_legacy_stream():
    """A cudaMemcpy from pageable memory may return before its data has landed, and it runs on
    the legacy stream, which non-blocking streams (all of torch's) do not wait for. Uploads go by
    cudaMemcpyAsync on the caller's stream. The drop-in functions run on the legacy stream
    throughout."""
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        if os.path.basename(path) == "dropin.cu":
            continue
        for call in re.findall(r"cudaMemcpy\s*\([^;]*;", open(path).read()):
            if "cudaMemcpyHostToDevice" in call:
                found.append((os.path.basename(path), " ".join(call.split())))
    assert not found, found


@pytest.mark.gpu
@pytest.mark.parametrize("n", [64, 75])
def test_used_at_once_on_a_side_stream(native, n):
    """Created and applied on a non-blocking stream without a wait in between: the values of an
    operator that has been waited for (planes of 128 and 150, own and library transforms)."""
    from lentils_gb300.operators import NUFFTOperator
    from lentils_gb300.spaces import ImageSpace, VisibilitySpace
    rng = np.random.default_rng(n)
    img = O.ImageGeom((n, n), [(-1.0, 1.0), (-1.0, 1.0)])
    padded, _, _ = O.padded_geom(img, 2)
    four = O.FourierGeom(padded)
    uvw = O.synth_uv(rng, 500, four, 0.4, 4)
    space, vis = ImageSpace((n, n), [(-1.0, 1.0), (-1.0, 1.0)]), VisibilitySpace([1.0], uvw)
    x = torch.as_tensor(rng.normal(size=(n, n))).cuda()
    want = NUFFTOperator(vis, space) * x
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        got = NUFFTOperator(vis, space) * x
    side.synchronize()
    assert O.rel_l2(got.cpu().numpy(), want.cpu().numpy()) < 1e-13
