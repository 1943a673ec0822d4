"""The precision form's separation from high and low FP32 parts, restated in numpy:
no further from the exact separation than the FP64 difference rounded to FP32, for
every pair that the kernels give to it (r above the guard times |x|, the guard
read from the source). Bars: the largest error within 2^-33 sqrt(3) r of the rounded
difference's (the parts leave out 2^-48 |x| per axis), the rms within 2^-12 of it."""
import os
import re

import numpy as np
import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "phantom_gb300", "csrc", "ph_walk.cuh")
F, D = np.float32, np.float64


def guard():
    m = re.search(r"const float m = ([0-9.e+-]+)f \* fmaxf\(fmaxf\(fabsf\(s\.h\.x\)", open(SRC).read())
    return float(m.group(1))


def parts(x):
    h = x.astype(F)
    return h, (x - h.astype(D)).astype(F)


def diff2(ah, al, bh, bl):
    s = ah - bh
    t = s - ah
    e = (ah - (s - t)) - (bh + t)
    return s + (e + (al - bl))


@pytest.mark.parametrize("octaves", [0, 1, 3, 6])
def test_error_of_the_two_float_separation(octaves):
    rng = np.random.default_rng(octaves)
    n = 300000
    x = rng.uniform(0.25, 1.0, (n, 3)) * rng.choice([-1, 1], (n, 3))
    d = rng.standard_normal((n, 3))
    d /= np.linalg.norm(d, axis=1)[:, None]
    y = x - d * (np.abs(x).max(1) * guard() * 2.0 ** octaves * rng.uniform(1, 2, n))[:, None]
    exact = x - y  # exact or rounded at 2^-53 of |x|
    new, old = diff2(*parts(x), *parts(y)), exact.astype(F)
    r = np.linalg.norm(exact, axis=1)
    en, eo = [np.linalg.norm(a.astype(D) - exact, axis=1) / r for a in (new, old)]
    assert en.max() <= eo.max() + 2.0 ** -33 * np.sqrt(3.0)
    assert abs(np.sqrt((en ** 2).mean()) / np.sqrt((eo ** 2).mean()) - 1.0) < 2.0 ** -12
