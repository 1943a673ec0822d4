"""The adjoint's j-side workspace where the force's lists sized it for fewer
values: lattices of a few hundred particles, and a context whose later particle
set has shorter lists than an earlier one. Gradients against the per-side pass,
within 1e-11 of their largest magnitude (both passes add the same few hundred
FP64 terms per particle, in different order)."""
import numpy as np
import pytest

from phantom_gb300 import capi
from phantom_gb300 import setups as S

pytestmark = pytest.mark.gpu


def case(n1d):
    cfg, x, v, B = S.hydro_lattice(n1d, jitter=0.2, seed=n1d)
    return dict(cfg, tolh=1.0e-8), x, v, B, np.random.default_rng(n1d).standard_normal((len(x), 4))


def gradients(ctx, x, v, B, w):
    ctx.upload(x, v, B)
    ctx.derivs(1, 0.0)
    return ctx.adjoint(w)


def per_side(n1d):
    cfg, x, v, B, w = case(n1d)
    ctx = capi.Context(cfg)
    ctx.set_tune(force_sym=0)
    return gradients(ctx, x, v, B, w)


def close(got, want):
    for a, b in zip(got, want):
        assert np.abs(a - b).max() <= 1.0e-11 * np.abs(b).max()


@pytest.mark.parametrize("n1d", [4, 5, 6, 7])
def test_small_lattice(n1d):
    cfg, x, v, B, w = case(n1d)
    close(gradients(capi.Context(cfg), x, v, B, w), per_side(n1d))


@pytest.mark.parametrize("sizes", [(12, 11), (12, 6, 12), (6, 13)])
def test_reused_context(sizes):
    sets = [case(n) for n in sizes]
    ctx = capi.Context(sets[0][0], maxp=max(len(s[1]) for s in sets))
    for n1d, (cfg, x, v, B, w) in zip(sizes, sets):
        ctx.set_params(cfg)
        close(gradients(ctx, x, v, B, w), per_side(n1d))
