"""Internal multipoles where the squared radius leaves FP32's normal numbers: next to the centre
(coordinates in radians put a pixel 1e-22 from a lens centre by rounding alone) and far out.

Tolerance: FP32 sums of up to 12 rotations (two roundings each) and two calls of powf (2 ulp):
(24 + 8) * 2^-24 = 2e-6 of the deflection."""
import numpy as np
import pytest
import torch

import oracle as O
from test_deflect_gpu import gpu_deflect

pytestmark = pytest.mark.gpu


def multipoles(pts, qh, coeff):
    d = pts[:, 0] + 1j * pts[:, 1]
    r, al = np.abs(d), 2.0 * qh
    e = d / r
    out = 0
    for i, (am, bm) in enumerate(coeff):
        m = i + 3
        em = e ** m
        norm = 2.0 / (m * m - (al - 2) ** 2) * r ** (1.0 - al)
        out = out + e * (-norm * (2.0 - al) * (bm * em.imag + am * em.real)
                         + 1j * norm * m * (-bm * em.real + am * em.imag))
    return np.stack([out.real, out.imag], 1)


@pytest.mark.parametrize("qh,nord", [(0.5, 2), (0.05, 1), (0.65, 4)])
@pytest.mark.parametrize("n", [1, 7, 64])
def test_near_and_far(native, qh, nord, n):
    rng = np.random.default_rng(n)
    coeff = rng.normal(0.0, 0.02, (nord, 2))
    lens = O.lens_array([O.multipole_cpars(0.0, 0.0, qh, 2 + nord, coeff)])
    r = 10.0 ** np.resize([-24, 0, -22, -20, 18.5, -19.2, -18.9, -18.8, 1, 19, 19.3, 20, 25, -5], n)
    th = rng.uniform(0, 2 * np.pi, n)
    pts = np.stack([r * np.cos(th), r * np.sin(th)], 1)
    want = multipoles(pts, qh, coeff)
    got = pts - gpu_deflect(lens, pts)
    err = np.hypot(*(got - want).T)
    size = np.hypot(*want.T)
    # the position itself is an FP64 number: its rounding, seen from the deflection
    assert (err <= 2e-6 * size + 2.0 ** -51 * r).all()
    near = r < 1
    p32 = pts.astype(np.float32).astype(np.float64)
    got = p32 - gpu_deflect(lens, p32, f32=True)
    assert np.isfinite(got).all()
    want = multipoles(p32[near], qh, coeff)
    err = np.hypot(*(got[near] - want).T)
    assert (err <= 3e-6 * np.hypot(*want.T) + 2.0 ** -23 * r[near]).all()


def test_centre(native):
    """At the centre itself the direction is undefined: NaN, as in the reference, and the other
    point of the pair is not touched. Without coefficients there is no deflection."""
    pts = np.array([[0.0, 0.0], [0.3, -0.2], [0.1, 0.4]])
    coeff = np.array([[0.01, 0.02]])
    for f32 in (False, True):
        got = gpu_deflect(O.lens_array([O.multipole_cpars(0.0, 0.0, 0.5, 3, coeff)]), pts, f32)
        assert np.isnan(got[0]).all() and np.isfinite(got[1:]).all()
        got = gpu_deflect(O.lens_array([O.multipole_cpars(0.0, 0.0, 0.5, 2, coeff[:0])]), pts, f32)
        assert np.array_equal(got, pts if not f32 else pts.astype(np.float32))
