"""Centre of mass of a node of 257 to 2048 particles: the reference adds the
particles one after the other, every partial sum rounded, and the block that
builds the subtree forms the same sum in integer arithmetic, 32 or 128 terms at
a time. Bit-identical to the literal loop where that arithmetic has to tell
cases apart: terms that are exact ties of the sum's last place, of both parities;
sums that change sign, leave their binade up or down, or stay zero; terms far
below the last place; and masses whose weight m (1/m) is not one."""
import numpy as np
import pytest

from phantom_gb300 import capi
from phantom_gb300 import setups as S

pytestmark = pytest.mark.gpu


def axis(kind, n, rng):
    i = np.arange(n)
    if kind == "ties":        # half of the last place once the sum is above 2, then quarters, ...
        return 1.0 + (2 * rng.integers(0, 8, n) + 1) * 2.0 ** -52
    if kind == "half":        # a large sum first, then halves of its last place with both signs
        return np.where(i < 3, 2.0 ** 30, rng.choice([-1.0, 1.0], n) * rng.integers(0, 4, n) * 2.0 ** -23)
    if kind == "negative":
        return -(1.0 + (2 * rng.integers(0, 8, n) + 1) * 2.0 ** -52)
    if kind == "cancel":      # crosses zero and its binades again and again
        return rng.standard_normal(n) * 2.0 ** rng.integers(-6, 6, n)
    if kind == "saw":         # up to a power of two and back, by steps that are ties there
        return np.where(i // 64 % 2 == 0, 1.0, -1.0) * (1.0 + 2.0 ** -45 * rng.integers(0, 2, n))
    if kind == "tiny":        # terms below the last place of the sum
        return np.where(i % 37 == 0, 1.0, 2.0 ** -60 * rng.integers(0, 5, n))
    if kind == "growing":
        return 2.0 ** (i % 300 / 8.0)
    if kind == "zeros":
        return np.where(i % 5 == 0, -0.0, 0.0)
    return rng.uniform(0.0, 1.0, n)


def centre(x, pm):
    dfac = 1.0 / pm
    fac = pm * dfac
    s, m = 0.0, 0.0
    for v in x.tolist():
        s = s + fac * v
        m = m + pm
    return s / (m * dfac)


PM_ONE = 1.0 / 512.0
PM_OTHER = next(p for p in (1.0 / k for k in range(3, 4000)) if p * (1.0 / p) != 1.0)


@pytest.mark.parametrize("pm", [PM_ONE, PM_OTHER])
@pytest.mark.parametrize("kinds", [("ties", "negative", "plain"), ("half", "cancel", "saw"), ("tiny", "growing", "plain"),
                                   ("zeros", "ties", "cancel")])
@pytest.mark.parametrize("n", [257, 288, 500, 1023, 2048])
def test_root_centre(n, kinds, pm):
    rng = np.random.default_rng(n)
    cfg, x, v, B = S.random_box(n, seed=n)
    cfg = dict(cfg, periodic=0, massoftype=pm)
    for a, k in enumerate(kinds):
        x[:, a] = axis(k, n, rng)
    ctx = capi.Context(cfg)
    ctx.upload(x, v, B)
    ctx.build_tree()
    t = ctx.nodes()
    root = np.flatnonzero(t["inoderange"][:, 1] - t["inoderange"][:, 0] == n - 1)
    assert len(root) == 1
    assert t["xcen"][root[0]].tolist() == [centre(x[:, a], pm) for a in range(3)]
