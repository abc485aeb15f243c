"""The reciprocal sum of the Ewald force field against a direct 64-bit sum over k vectors,
at the edges of the device passes: columns of four nz (kmax 3, 4, 7, 8), tiles of 32 and
blocks of 128 sites, oblong boxes.

Tolerance: every term of the sums is a product of three factors built by at most kmax
complex multiplications (about 4 eps each), so an output is off by less than
(16 kmax + 64) eps times the sum of its terms' magnitudes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def direct(pos, box, q, alpha, kmax, coulomb):
    n = np.stack(np.meshgrid(*[np.arange(-kmax, kmax + 1)] * 3, indexing="ij"), -1).reshape(-1, 3)
    n2 = (n * n).sum(1)
    n = n[(n2 > 0) & (n2 < kmax * kmax + 2)]
    k = 2 * np.pi * n / box
    k2 = (k * k).sum(1)
    f = coulomb * 2 * np.pi / np.prod(box) * np.exp(-k2 / (4 * alpha ** 2)) / k2
    phase = pos @ k.T
    s = q @ np.exp(1j * phase)
    u = 2 * f * (np.cos(phase) * s.real + np.sin(phase) * s.imag)
    g = 2 * f * (np.sin(phase) * s.real - np.cos(phase) * s.imag)
    mag = 2 * f * np.abs(q).sum()
    return (np.sum(f * np.abs(s) ** 2), np.sum(f) * np.abs(q).sum() ** 2, u.sum(1), mag.sum(),
            q[:, None] * (g @ k), np.abs(q)[:, None] * (mag @ np.abs(k)))


@pytest.mark.parametrize("kmax", [1, 3, 4, 7, 8, 13])
@pytest.mark.parametrize("n", [1, 31, 33, 129, 700])
def test_reciprocal_sum_matches_direct_sum(md, n, kmax):
    rng = np.random.default_rng(100 * n + kmax)
    box = np.array([9.0, 11.5, 14.0])
    pos = (rng.random((n, 3)) - 0.5) * box
    q = rng.normal(size=n)
    alpha, rc = 0.45, 2.0
    s = md.System.from_arrays(pos, box, charge=q, mol=np.arange(n))
    with_k, without = md.Ewald(rc, kmax, alpha, skin=0.5), md.Ewald(rc, 0, alpha, skin=0.5)
    e, e_mag, u, u_mag, f, f_mag = direct(pos, box, q, alpha, kmax, md.coulomb_prefactor())
    tol = (16 * kmax + 64) * EPS
    assert without.compute_forces(s)["reciprocal"] == 0.0
    f0, u0 = s.forces, without.charge_gradient(s)
    assert abs(with_k.compute_forces(s)["reciprocal"] - e) <= tol * e_mag
    # the other terms are common to both evaluations; adding them rounds once more
    got = s.forces - f0
    assert np.all(np.abs(got - f) <= tol * f_mag + 4 * EPS * np.abs(f0))
    assert np.all(np.abs(with_k.charge_gradient(s) - u0 - u) <= tol * u_mag + 4 * EPS * np.abs(u0))
