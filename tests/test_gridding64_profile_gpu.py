"""The paired-FP32 operators (csrc/gridding64.cu) against sums with the Kaiser-Bessel profile itself,
for every width they take: what a user sees, fit and rounding together.

Tolerance. The degree-11 fits are within FIT of the profile's peak at beta = 2.34 (2w) (12 Chebyshev
nodes per tap, evaluated in FP64). Seen from the rms weight of an axis that is FIT * peak / rms, on
each of two axes; the pairs' own rounding is the 7e-13 of the tests against the same fits."""
import numpy as np
import pytest

import oracle as O
import test_gridding64_gpu as G

pytestmark = pytest.mark.gpu
FIT = {1: 4.0e-10, 2: 4.1e-11, 3: 4.7e-12, 4: 4.6e-13}


def profile(f, w, beta, n):
    a = (f + w - 1 - np.arange(2 * w)[:, None]) / w
    return np.i0(beta * np.sqrt(np.maximum(0.0, 1 - a * a))) / (2 * w)


@pytest.mark.parametrize("tile", [8, 16])
@pytest.mark.parametrize("w", [1, 2, 3, 4])
def test_against_the_profile(native, monkeypatch, w, tile):
    monkeypatch.setattr(G, "weights", profile)
    rng = np.random.default_rng(w)
    four, ref, plan = G.setup(rng, 96, 75, w, 4000, tile)
    grid, vis = G.cnormal(rng, four.nu, four.half_nv), G.cnormal(rng, 4000)
    wt = profile(np.linspace(0, 1, 257), w, 2.34 * 2 * w, 0)
    tol = 2 * FIT[w] * wt.max() / np.sqrt((wt ** 2).mean()) + G.TOL
    y, g = G.both(plan, four, grid, vis)
    assert O.rel_l2(y, ref.degrid(grid)) < tol
    assert O.rel_l2(g, ref.grid(vis)) < tol
