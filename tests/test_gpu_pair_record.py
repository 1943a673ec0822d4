"""The precision form's pair record where its buffer has to grow: a context that
has recorded a set of few neighbours steps one of many. The step must equal,
bit for bit, that of a fresh context, which records the same pairs after sweeping
its first evaluations."""
import numpy as np
import pytest

from phantom_gb300 import capi
from phantom_gb300 import setups as S

pytestmark = pytest.mark.gpu


def state(ctx, x, v, B, dt=None):
    ctx.upload(x, v, B)
    dt = dt or ctx.derivs(1, 0.0)
    r = ctx.step(0.0, dt)
    n = len(x)
    out = [np.zeros((n, 4)) for _ in range(5)] + [np.zeros(n, np.float32)]
    ctx.download_state(*out)
    return r, out


@pytest.mark.parametrize("n1d", [8, 20, 44])
@pytest.mark.parametrize("mk", [S.hydro_lattice, S.mhd_vortex])
def test_record_grows(n1d, mk):
    small, large = [mk(n1d, jitter=0.2, seed=3, hfact=hf) for hf in (1.0, 1.5)]
    cfgs = [dict(c[0], tolv=1.0e-8) for c in (small, large)]
    warm = capi.Context(cfgs[0], precision=capi.PH_PREC_MIXED)
    for _ in range(2):
        warm.upload(*small[1:])
        assert warm.step(0.0, warm.derivs(1, 0.0))[1] >= 3
    warm.set_params(cfgs[1])
    fresh = capi.Context(cfgs[1], precision=capi.PH_PREC_MIXED)
    for _ in range(2):  # the step that grows the record, then one that replays from its second evaluation
        got, want = [state(c, *large[1:]) for c in (warm, fresh)]
        assert got[0] == want[0] and got[0][1] >= 3
        for a, b in zip(got[1], want[1]):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("mk", [S.hydro_lattice, S.mhd_vortex])
def test_record_limits(mk):
    """No record, one that does not fit, one given up between steps and one that
    is bounded but fits: the same steps, bit for bit."""
    cfg, x, v, B = mk(16, jitter=0.2, seed=3)
    cfg = dict(cfg, tolv=1.0e-8)
    n = len(x)
    runs = []
    for limits in ((-1, -1, -1), (0, 0, 0), (4096, 4096, 4096), (-1, 4096, -1), (0, 1 << 30, 1 << 30)):
        ctx = capi.Context(cfg, precision=capi.PH_PREC_MIXED)
        ctx.upload(x, v, B)
        dt, out = ctx.derivs(1, 0.0), []
        for lim in limits:
            ctx.set_record_limit(lim)
            r = ctx.step(0.0, dt)
            assert r[1] >= 3
            out.append(r)
        out += list(ctx.download())
        runs.append(out)
    for run in runs[1:]:
        for a, b in zip(run, runs[0]):
            assert np.array_equal(a, b)
