"""The tile and the work-item size that a plan chooses by itself: by kernel width, grid and number
of visibilities (csrc/plan.cu; the measurements stand there)."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,n,nvis,tile,chunk", [
    (3, 128, 20000, 8, 66), (4, 256, 500000, 8, 1024), (4, 512, 10000, 8, 64),
    (4, 690, 300000, 8, 1000), (4, 690, 20000, 16, 256), (2, 720, 40000, 16, 256),
    (4, 1024, 100000, 16, 256), (3, 1024, 200000, 16, 400), (4, 1024, 2000000, 16, 3289),
    (5, 256, 131072, 8, 256), (6, 512, 500000, 8, 625), (6, 256, 30000, 16, 256), (6, 65, 600000, 16, 986),
    (6, 690, 500000, 16, 822), (8, 128, 20000, 16, 256), (8, 340, 300000, 16, 493)])
def test_defaults(native, w, n, nvis, tile, chunk):
    from lentils_gb300.gridding import GriddingPlan
    rng = np.random.default_rng(w)
    img = O.ImageGeom((n, n), [(-1.0, 1.0), (-1.0, 1.0)])
    four = O.FourierGeom(img)
    uvw = O.synth_uv(rng, nvis, four, 0.45, w)
    stats = GriddingPlan(uvw, [1.0], four.nu, four.nv, four.du, four.dv, 0.0, 0.0, w,
                         2.34 * 2 * w).stats
    assert stats["tile"] == tile
    assert stats["max_item_vis"] <= chunk
    if stats["heaviest_tile_vis"] > chunk:
        assert stats["max_item_vis"] == chunk
