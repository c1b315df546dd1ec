"""The paired-FP32 gridding (csrc/gridding64.cu) cell by cell: a strong visibility has no part in
the rounding of grid cells that its window does not cover, whatever its place in the sort order.

Tolerance. The visibilities of one cell are summed with a bias below 4 (2w) times the largest
term, and the low halves of a sum lose at most 2^-45 of the bound per term: for up to 8 terms a
batch, 8 * 32 * 2^-45 = 7.3e-12 of the largest product of a weight and a visibility that reaches
the cell; 1e-11 with the weights' own rounding."""
import numpy as np
import pytest

from test_gridding64_gpu import both, cnormal, setup

pytestmark = pytest.mark.gpu


def reach(ref, four, mag):
    """Per half-plane cell, the largest |visibility| whose window covers it."""
    out = np.zeros((four.nu, four.nv))
    for u, v, k in ref._cells():
        np.maximum.at(out, (u, v), np.where(k != 0, mag, 0.0))
    half = out[:, :four.half_nv].copy()
    mir = np.roll(np.flip(out, (0, 1)), (1, 1), (0, 1))
    top = four.nv - four.half_nv
    half[:, 1:top + 1] = np.maximum(half[:, 1:top + 1], mir[:, 1:top + 1])
    return half


@pytest.mark.parametrize("ratio", [1e-4, 1e-8, 1e-14])
@pytest.mark.parametrize("w,tile,nx,ny,nvis,chunk", [
    (1, 16, 64, 64, 900, 0), (2, 16, 96, 80, 700, 0), (3, 8, 120, 100, 500, 4096),
    (3, 16, 128, 96, 400, 0), (4, 16, 192, 160, 500, 4096), (4, 8, 160, 128, 300, 0)])
def test_weak_next_to_strong(native, w, tile, nx, ny, nvis, chunk, ratio):
    rng = np.random.default_rng(int(-np.log10(ratio)) + 10 * w + tile)
    four, ref, plan = setup(rng, nx, ny, w, nvis, tile, 0, chunk)
    vis = cnormal(rng, nvis)
    vis[rng.random(nvis) < 0.8] *= ratio
    _, got = both(plan, four, np.zeros((four.nu, four.half_nv), complex), vis)
    want, size = ref.grid(vis), reach(ref, four, np.abs(vis))
    peak = (np.i0(2.34 * 2 * w) / (2 * w)) ** 2
    weak = (size > 0) & (size < 1e3 * ratio) & (size < 0.1)
    assert weak.sum() > 50
    assert (np.abs(got - want)[size > 0] < 1e-11 * peak * size[size > 0]).all()
    assert (got[size == 0] == 0).all()


@pytest.mark.parametrize("ratio", [1e-30, 1e-150, 1e-312])
@pytest.mark.parametrize("w,tile,nx,ny,nvis,integer", [
    (1, 16, 64, 64, 900, 30), (2, 8, 96, 80, 700, 0), (3, 16, 128, 96, 400, 40),
    (4, 16, 192, 160, 500, 60)])
def test_beyond_the_range_of_pairs(native, w, tile, nx, ny, nvis, integer, ratio):
    """Values that FP64 holds side by side and pairs of FP32 values do not (2^-77 of the largest of
    a work item and below, subnormals): gridded and degridded to the same tolerance, relative to
    what reaches each result."""
    rng = np.random.default_rng(int(-np.log10(ratio)) + 10 * w + tile)
    four, ref, plan = setup(rng, nx, ny, w, nvis, tile, integer)
    peak = (np.i0(2.34 * 2 * w) / (2 * w)) ** 2
    vis = cnormal(rng, nvis)
    vis[rng.random(nvis) < 0.7] *= ratio
    half = rng.random(nvis) < 0.3  # parts of one value may be far apart too
    vis[half] = vis[half].real + 1j * (ratio * vis[half].imag)
    grid = cnormal(rng, four.nu, four.half_nv)
    grid[:, four.half_nv // 3:] *= ratio
    y, g = both(plan, four, grid, vis)
    for part, pick in ((vis.real, np.real), (vis.imag, np.imag)):
        want, size = pick(ref.grid(part if pick is np.real else 1j * part)), reach(ref, four, np.abs(part))
        ok = size > 0
        assert (np.abs(pick(g) - want)[ok] <= 1e-11 * peak * size[ok]).all()
    full = np.zeros((four.nu, four.nv), complex)
    full[:, :four.half_nv] = grid
    mir = np.roll(np.flip(full, (0, 1)), (1, 1), (0, 1)).conj()
    full[:, four.half_nv:] = mir[:, four.half_nv:]
    want = ref.degrid(grid)
    for pick in (np.real, np.imag):
        size = np.zeros(nvis)
        for u, v, k in ref._cells():
            size = np.maximum(size, np.where(k != 0, np.abs(pick(full[u, v])), 0.0))
        assert (size < 1e3 * ratio).sum() > 10
        assert (np.abs(pick(y) - pick(want)) <= 1e-11 * peak * size).all()
