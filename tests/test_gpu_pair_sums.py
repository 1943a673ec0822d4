"""FP64 pair sums against all-pairs numpy sums at the places where the pair
kernels switch branch: neighbours at exactly two smoothing lengths, the knot of
the spline at one, coincident particles, the periodic wrap, and the softened
and 1/r^2 parts of self-gravity."""
import numpy as np
import pytest

from phantom_gb300 import capi, setups

pytestmark = pytest.mark.gpu
LD = np.longdouble
PI_REF = LD(3.1415926536)


def separations(cfg, x):
    d = x[:, None, :] - x[None, :, :]
    if cfg["periodic"]:
        for a, (lo, hi) in enumerate((("xmin", "xmax"), ("ymin", "ymax"), ("zmin", "zmax"))):
            L = cfg[hi] - cfg[lo]
            d[..., a] = np.where(np.abs(d[..., a]) > 0.5 * L, d[..., a] - np.copysign(L, d[..., a]), d[..., a])
    return d


def spline(q):
    w = np.where(q < 1, 1 - 1.5 * q ** 2 + 0.75 * q ** 3, np.where(q < 2, 0.25 * (2 - q) ** 3, 0))
    g = np.where(q < 1, q * (2.25 * q - 3), np.where(q < 2, -0.75 * (2 - q) ** 2, 0))
    return w, g


def dphidh(q):
    return np.where(q < 1, -0.6 * q ** 5 + 1.5 * q ** 4 - 2 * q ** 2 + 1.4,
                    np.where(q < 2, 0.2 * q ** 5 - 1.5 * q ** 4 + 4 * q ** 3 - 4 * q ** 2 + 1.6, 0))


@pytest.mark.parametrize("ulps", [-2, -1, 0, 1, 2])
@pytest.mark.parametrize("dist2", [1, 2, 3, 4])
def test_neighbours_at_the_kernel_edge(ulps, dist2):
    """h = dist/2 within a few ulps: the neighbours at that distance are in or
    out as the reference's r^2 h^-2 < 4 rounds."""
    cfg, x, v, B = setups.exact_lattice(8)
    h = np.float64(0.5 * np.sqrt(dist2 / 64.0))
    for _ in range(abs(ulps)):
        h = np.nextafter(h, np.inf if ulps > 0 else 0.0)
    x[:, 3] = h
    d = separations(cfg, x[:, :3])
    r2 = d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1] + d[..., 2] * d[..., 2]
    h1 = 1.0 / h
    want = (r2 * (h1 * h1) < 4.0).sum(1)  # the particle itself included
    ctx = capi.Context(cfg)
    ctx.upload(x, v, B)
    ctx.build_tree()
    got = ctx.densityiterate(0)["nneigh"]
    assert np.array_equal(got, want)


@pytest.mark.parametrize("case", ["lattice", "open", "gravity", "coincident", "knot"])
def test_density_sums(case):
    """rho, 1/Omega and gradsoft of one pass at the given h. Each pair term
    takes fewer than 16 roundings and at most 140 terms are added: rho is
    within 160 x 2^-53 of the exact sum (h = hfact (m/rho)^(1/3) within a third
    of it, plus the cube root); 1/Omega and gradsoft are stored in float32,
    and cancel at most an order of magnitude."""
    if case in ("lattice", "knot", "coincident"):
        cfg, x, v, B = setups.hydro_lattice(9, jitter=0.0 if case == "knot" else 0.2, seed=4)
        if case == "knot":
            x[:, 3] = 1.0 / 9.0  # neighbours at q = 1 to rounding
        if case == "coincident":
            x[10, :3] = x[11, :3]
    else:
        cfg, x, v, B = setups.random_box(600, seed=5, gravity=case == "gravity")
    h = x[:, 3].copy()
    ctx = capi.Context(cfg)
    ctx.upload(x, v, B)
    xw, perm, _ = ctx.build_tree()
    d = ctx.densityiterate(0)
    m, hl = LD(cfg["massoftype"]), h.astype(LD)
    s = separations(cfg, xw[:, :3]).astype(LD)
    q = np.sqrt((s * s).sum(-1)) / hl[:, None]
    w, g = spline(q)
    rho = m * w.sum(1) / PI_REF / hl ** 3
    grad = m * (-q * g - 3 * w).sum(1) / PI_REF / hl ** 4
    dh = -hl / (3 * m * (LD(cfg["hfact"]) / hl) ** 3)
    want_h = LD(cfg["hfact"]) * (m / rho) ** (LD(1) / 3)
    assert np.abs(d["xyzh"][:, 3] / want_h - 1).max() < 160 * 2.0 ** -53
    om = 1 - dh * grad
    assert np.abs(d["gradh"][:, 0] * om - 1).max() < 2.0 ** -22
    if case == "gravity":
        gs = m * dphidh(q).sum(1) / hl ** 2 * dh
        assert np.abs(d["gradh"][:, 1] - gs).max() < 2.0 ** -22 * np.abs(gs).max()


@pytest.mark.parametrize("gap", [1e-4, 3e-6, 2e-7, 1e-9, 1e-13])
@pytest.mark.parametrize("shift", [0.0, 0.49])
def test_mixed_separation_of_close_pairs(gap, shift):
    """Precision form: pairs far closer than the coordinates' FP32 rounding, in
    the box and across its face, keep the direction and size of their FP64
    separation: one derivs against the plain form, within the form's 1e-5."""
    cfg, x, v, B = setups.hydro_lattice(12, jitter=0.1, seed=6)
    rng = np.random.default_rng(7)
    pick = rng.choice(len(x), 40, replace=False)
    d = rng.standard_normal((20, 3))
    x[pick[20:], :3] = x[pick[:20], :3] + gap * d / np.linalg.norm(d, axis=1)[:, None]
    x[:, :3] = np.mod(x[:, :3] + shift, 1.0)
    out = []
    for prec in (capi.PH_PREC_FP64, capi.PH_PREC_MIXED):
        ctx = capi.Context(dict(cfg, tolh=1e-7), precision=prec)
        ctx.upload(x, v, B)
        ctx.build_tree()
        h = ctx.densityiterate(1)["xyzh"][:, 3]
        out.append((h, ctx.force(1, 0.0)["fxyzu"]))
    assert np.abs(out[1][0] / out[0][0] - 1).max() < 1e-6
    for c in (slice(0, 3), 3):
        assert np.abs(out[1][1][:, c] - out[0][1][:, c]).max() < 1e-5 * np.abs(out[0][1][:, c]).max()
