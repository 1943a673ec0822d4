"""A context whose parameters change between a force and the next: the trial
lists, with the owned entries' offsets of the symmetric pair pass, belong to
the parameters that they were made with. Bars: the symmetric pass within 1e-12 of the
per-side pass on the same density, its gradients within 1e-11."""
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


@pytest.mark.parametrize("setup", ["hydro", "mhd"])
@pytest.mark.parametrize("earlier", [False, True])
def test_lists_of_the_plain_form(setup, earlier):
    cfg, x, v, B = case(setup)
    if earlier:  # offsets of other lists in the context
        ctx = solved(*case(setup, seed=6), FP64)
        ctx.force(1, 0.0)
        ctx.set_params({}, MIXED)
        ctx.upload(x, v, B)
        ctx.build_tree()
        ctx.densityiterate(1)
    else:
        ctx = solved(cfg, x, v, B, MIXED)
    ctx.force(1, 0.0)
    ctx.set_params({}, FP64)
    got = ctx.force(1, 0.0)
    w = np.random.default_rng(1).standard_normal((len(x), 4))
    grad = ctx.adjoint(w)[:2] if setup == "hydro" else ()
    ctx.set_tune(force_sym=0)
    want = ctx.force(1, 0.0)
    close(got["fxyzu"], want["fxyzu"], 1.0e-12)
    if setup == "mhd":
        close(got["dBevol"], want["dBevol"], 1.0e-12)
    else:
        for a, b in zip(grad, ctx.adjoint(w)[:2]):
            close(a, b, 1.0e-11)


def test_hydro_lists_then_mhd():
    """Switching the magnetic field on adds values to the symmetric pass's rows."""
    cfg, x, v, B = case("mhd")
    ctx = solved(dict(cfg, mhd=0), x, v, B, FP64)
    ctx.force(1, 0.0)
    ctx.set_params(dict(mhd=1))
    got = ctx.force(1, 0.0)
    ctx.set_tune(force_sym=0)
    want = ctx.force(1, 0.0)
    close(got["fxyzu"], want["fxyzu"], 1.0e-12)
    close(got["dBevol"], want["dBevol"], 1.0e-12)


def test_self_gravity_needs_its_own_tree():
    """A tree and density made without self-gravity have no quadrupoles and no
    softening sums."""
    cfg, x, v, B = case("cloud")
    ctx = solved(dict(cfg, gravity=0), x, v, B, FP64)
    ctx.set_params(dict(gravity=1))
    with pytest.raises(capi.PhantomError) as e:
        ctx.force(1, 0.0)
    assert e.value.code == 13
    with pytest.raises(capi.PhantomError) as e:
        ctx.densityiterate(1)
    assert e.value.code == 13
    ctx.upload(x, v, B)  # the given h again: the tree's hmax, hence its opening, depends on it
    ctx.build_tree()
    ctx.densityiterate(1)
    got = ctx.force(1, 0.0)["fxyzu"]
    close(got[:, :3], solved(cfg, x, v, B, FP64).force(1, 0.0)["fxyzu"][:, :3], 1.0e-9)


def test_self_gravity_switched_on_before_a_step():
    """The step kicks with the forces it has and evaluates with its own tree: as
    from the same state uploaded into a context with self-gravity."""
    cfg, x, v, B = case("cloud")
    ctx = capi.Context(dict(cfg, gravity=0))
    ctx.upload(x, v, B)
    dt = ctx.derivs(1, 0.0)
    n = len(x)
    st = [np.zeros((n, 4)) for _ in range(5)] + [np.zeros(n, np.float32)]
    ctx.download_state(*st)
    ctx.set_params(dict(gravity=1))
    want = capi.Context(cfg)
    want.upload_state(*st)
    assert ctx.step(0.0, dt) == want.step(0.0, dt)
    for a, b in zip(ctx.download(), want.download()):
        assert np.array_equal(a, b)
