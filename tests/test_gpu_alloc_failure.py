"""A request that no device has room for (checkpoints of four million steps, one
allocation of 690 GB that is refused at once) returns its status and leaves the
context as it was: no pending CUDA error for the next launch check, and steps
that give the same bits, the pair record they replay having been given up."""
import numpy as np
import pytest

from phantom_gb300 import capi
from phantom_gb300 import setups as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [capi.PH_PREC_MIXED, capi.PH_PREC_FP64])
def test_refused_allocation(precision):
    cfg, x, v, B = S.hydro_lattice(12, jitter=0.2, seed=3)
    cfg = dict(cfg, tolv=1.0e-8)
    out = []
    for refuse in (True, False):
        ctx = capi.Context(cfg, precision=precision)
        ctx.upload(x, v, B)
        dt = ctx.derivs(1, 0.0)
        r = [ctx.step(0.0, dt) for _ in range(2)]
        assert r[0][1] >= 3
        if refuse:
            with pytest.raises(capi.PhantomError) as e:
                ctx.rollout_adjoint(np.full(4000000, 1.0e-4), np.ones((len(x), 4)), 1)
            assert e.value.code == 2
        r += [ctx.step(0.0, dt) for _ in range(2)]
        ctx.build_tree()
        ctx.densityiterate(1)
        out.append(r + list(ctx.download()))
    for a, b in zip(*out):
        assert np.array_equal(a, b)
