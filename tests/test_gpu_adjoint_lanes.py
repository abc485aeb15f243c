"""The adjoint's pair pass at rows shorter and longer than its eight lanes and at block
remainders: the Hessian-vector product and parameter derivatives against a direct 64-bit
sum.  Tolerance: some forty operations a pair, so 100 eps of the terms' magnitudes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


def direct(pos, box, mu, rc, lfs):
    d = pos[:, None] - pos[None]
    d -= box * np.round(d / box)
    s = (d * d).sum(-1)
    np.fill_diagonal(s, 1e9)
    on = s < rc * rc
    s = np.where(on, s, 1.0)
    t3 = s ** -3.0
    w = 24 * (2 * t3 * t3 - t3)
    w_s = 24 * (-12 * t3 * t3 + 3 * t3) / s
    w_sig = 24 * (24 * t3 * t3 - 6 * t3)
    if lfs:
        c3 = rc ** -6.0
        r = np.sqrt(s)
        slope, slope_sig = -24 * (2 * c3 * c3 - c3) / rc, -24 * (24 * c3 * c3 - 6 * c3) / rc
        w, w_s, w_sig = w + r * slope, w_s + 0.5 * slope / r, w_sig + r * slope_sig
    g, g_s, g_sig = [np.where(on, x, 0.0) for x in (w / s, (w_s - w / s) / s, w_sig / s)]
    a = mu[:, None] - mu[None]
    dm = (d * a).sum(-1)
    h = (g[..., None] * a + (2 * g_s * dm)[..., None] * d).sum(1)
    h_mag = (np.abs(g[..., None] * a) + np.abs(2 * g_s[..., None] * d) * (np.abs(d * a)).sum(-1)[..., None]).sum(1)
    f, f_sig = (g[..., None] * d).sum(1), (g_sig[..., None] * d).sum(1)
    mags = [(np.abs(mu)[:, None] * np.abs(k[..., None] * d)).sum() for k in (g, g_sig)]
    return h, h_mag, (mu * f).sum(), (mu * f_sig).sum(), mags


@pytest.mark.parametrize("lfs", [0, 1])
@pytest.mark.parametrize("n", [2, 7, 9, 33, 257, 700])
def test_hvp_matches_direct_sum(md, n, lfs):
    rng = np.random.default_rng(n)
    side = int(np.ceil(n ** (1 / 3)))
    box = np.array([9.0, 9.6, 10.2])
    cell = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    pos = (cell + 0.5) * (box / max(side, 9)) - 0.5 * box + rng.uniform(-0.05, 0.05, (n, 3))
    mu = rng.normal(size=(n, 3))
    s = md.System.from_arrays(pos, box, mass=np.ones(n))
    v = md.VerletList(box, 2.5, 0.3)
    v.build(s)
    h, th = md.LennardJones(1.0, 1.0, 2.5, lfs).hessian_vector_product(s, v, mu)
    ref, mag, te, ts, (me, ms) = direct(pos, box, mu, 2.5, lfs)
    assert np.all(np.abs(h - ref) <= 100 * EPS * (1 + mag))
    assert abs(th[0] - te) <= 100 * EPS * (1 + me) and abs(th[1] - ts) <= 100 * EPS * (1 + ms)
