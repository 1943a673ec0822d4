"""A context whose precision changes between the density and what follows it.

The precision form's force and adjoint need the low parts of the positions, which
the plain form's density has no use for. Sets lie 64 box lengths off the origin,
where a position's FP32 part is 1e-4 of a particle separation away from it, so
that a missing low part shows. Bars: the precision form within 1e-5 of the plain
form's largest value (its target), its gradients within 1e-4."""
import numpy as np
import pytest

from phantom_gb300 import capi
from phantom_gb300 import setups as S

pytestmark = pytest.mark.gpu
FP64, MIXED = capi.PH_PREC_FP64, capi.PH_PREC_MIXED


def case(setup, seed=5):
    if setup == "cloud":
        cfg, x, v, B = S.gravity_cloud(3000, seed=seed)
    else:
        cfg, x, v, B = (S.mhd_vortex if setup == "mhd" else S.hydro_lattice)(14, jitter=0.2, seed=seed)
        cfg["periodic"] = 0
    x[:, :3] += 64.0
    return dict(cfg, tolh=1.0e-7), x, v, B


def solved(cfg, x, v, B, precision):
    ctx = capi.Context(cfg, precision=precision)
    ctx.upload(x, v, B)
    ctx.build_tree()
    ctx.densityiterate(1)
    return ctx


def close(a, b, tol):
    assert np.abs(a - b).max() <= tol * np.abs(b).max()


@pytest.mark.parametrize("earlier", [False, True])
@pytest.mark.parametrize("setup", ["hydro", "mhd", "cloud"])
def test_low_words_of_the_force(setup, earlier):
    cfg, x, v, B = case(setup)
    want = solved(cfg, x, v, B, FP64).force(1, 0.0)
    if earlier:  # low parts of another set in the context
        ctx = solved(*case(setup, seed=6), MIXED)
        ctx.set_params({}, FP64)
        ctx.upload(x, v, B)
        ctx.build_tree()
        ctx.densityiterate(1)
    else:
        ctx = solved(cfg, x, v, B, FP64)
    ctx.set_params({}, MIXED)
    got = ctx.force(1, 0.0)
    close(got["fxyzu"][:, :3], want["fxyzu"][:, :3], 1.0e-5)
    if setup == "mhd":
        close(got["dBevol"][:, :3], want["dBevol"][:, :3], 1.0e-5)


def test_low_words_of_the_adjoint():
    cfg, x, v, B = case("hydro")
    w = np.random.default_rng(1).standard_normal((len(x), 4))
    want = solved(cfg, x, v, B, FP64).adjoint(w)
    ctx = solved(cfg, x, v, B, FP64)
    ctx.set_params({}, MIXED)
    for a, b in zip(ctx.adjoint(w), want):
        close(a, b, 1.0e-4)


def test_low_words_after_a_refit():
    cfg, x, v, B = case("hydro")
    ctx = solved(cfg, x, v, B, MIXED)
    x = x + np.array([0.37, -0.21, 0.11, 0.0])
    out = []
    for precision in (FP64, MIXED):
        ctx.set_params({}, FP64)
        ctx.revtree(x)
        ctx.densityiterate(1)
        ctx.set_params({}, precision)
        out.append(ctx.force(1, 0.0)["fxyzu"])
    close(out[1][:, :3], out[0][:, :3], 1.0e-5)
