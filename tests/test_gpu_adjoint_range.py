"""The precision form's hydro adjoint at densities whose squares leave the FP32
range. Accelerations and du/dt, and so their gradients, do not change when every
particle mass is multiplied by one factor (u, h and positions kept), and a power
of two scales every product exactly: gradients within 1e-6 of their largest value
(FP32 rounding times an order of magnitude for the sums)."""
import numpy as np
import pytest

from phantom_gb300 import capi
from phantom_gb300 import setups as S

pytestmark = pytest.mark.gpu


def gradients(cfg, x, v, B, w, scale):
    ctx = capi.Context(dict(cfg, massoftype=cfg["massoftype"] * scale, tolh=1.0e-6), precision=capi.PH_PREC_MIXED)
    ctx.upload(x, v, B)
    return ctx.adjoint(w)


@pytest.mark.parametrize("cond", [True, False])
@pytest.mark.parametrize("exponent", [-40, -60, -66, -80, 20])
def test_gradients_do_not_depend_on_the_mass_unit(exponent, cond):
    cfg, x, v, B = S.hydro_lattice(12, jitter=0.2, seed=8)
    v[:, 3] *= 1.0 + 0.3 * np.sin(2.0 * np.pi * x[:, 0])  # pressure differences for the conductivity
    if not cond:
        cfg["alphau"] = 0.0
    w = np.random.default_rng(2).standard_normal((len(x), 4))
    want = gradients(cfg, x, v, B, w, 1.0)
    got = gradients(cfg, x, v, B, w, 2.0 ** exponent)
    for a, b in zip(got, want):
        assert np.abs(a - b).max() <= 1.0e-6 * np.abs(b).max()
