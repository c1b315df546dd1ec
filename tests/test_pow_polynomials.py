"""The fits inside pow_pos (csrc/deflect_device.cuh), with the coefficients as they stand in the
source, FP32 values, evaluated in FP64: the errors that the comment beside them states."""
import os
import re

import numpy as np

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lentils_gb300",
                   "csrc", "deflect_device.cuh")


def coefficients(body, name):
    """Leading coefficient first: `name = splat(c)` and the ffma2 steps after it."""
    first = re.search(r"float2 %s = splat\((.*?)f\);" % name, body).group(1)
    rest = re.findall(r"%s = __ffma2_rn\(%s, \w, splat\((.*?)f\)\);" % (name, name), body)
    c = [np.float32(v) for v in [first] + rest]
    return np.array(c, dtype=np.float64)


def test_fits_of_the_power():
    body = open(SRC).read().split("float2 pow_pos(", 1)[1].split("\n}", 1)[0]
    p, r = coefficients(body, "p"), coefficients(body, "r")
    assert len(p) == 10 and len(r) == 7
    f = np.linspace(np.sqrt(0.5) - 1, np.sqrt(2.0) - 1, 200001)
    assert np.abs(np.polyval(p, f) * f - np.log2(1 + f)).max() < 1.6e-9
    y = np.linspace(-0.5, 0.5, 200001)
    assert np.abs(np.polyval(r, y) / 2.0 ** y - 1).max() < 3.1e-9
