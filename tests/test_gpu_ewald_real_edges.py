"""The real-space pass at its edges: sizes around a block and around the changes of threads
per site, sites much closer than the shared reciprocals' range, against a direct 64-bit sum.

Tolerance: a term is a handful of FP64 operations and one erfc and exp (2 ulp each in CUDA's
tables), below 64 eps; the sums add at most 1e3 terms, so 1e-12 of the sum of magnitudes."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def direct(pos, box, q, mol, rc, alpha, c):
    d = pos[:, None] - pos[None]
    d -= box * np.round(d / box)
    r2 = (d * d).sum(-1)
    pair = (r2 < rc * rc) & (mol[:, None] != mol[None])
    r = np.sqrt(np.where(pair, r2, 1.0))
    erfc = np.vectorize(math.erfc)(alpha * r)
    cqq = c * q[:, None] * q[None]
    w = np.where(pair, cqq * (2 * alpha / math.sqrt(math.pi) * np.exp(-(alpha * r) ** 2) + erfc / r), 0.0)
    e = np.where(pair, cqq * erfc / r, 0.0)
    f = (w / r ** 2)[..., None] * d
    return e.sum() / 2, np.abs(e).sum(), f.sum(1), np.abs(f).sum(1)


@pytest.mark.parametrize("n", [1, 3, 4, 63, 65, 333, 1500])
def test_real_space_matches_direct_sum(md, n):
    rng = np.random.default_rng(n)
    box = np.array([14.0, 15.0, 17.0])
    pos = (rng.random((n, 3)) - 0.5) * box
    if n > 3:  # far below the range of the shared reciprocals, still representable
        pos[0], pos[1] = [0.0, 0.0, 0.0], [1e-9, 0.0, 0.0]
    q, mol = rng.normal(size=n), np.arange(n) // 2
    mol[:2] = [n, n + 1][:n]
    s = md.System.from_arrays(pos, box, charge=q, mol=mol)
    rc, alpha = 4.5, 0.6
    ew = md.Ewald(rc, 0, alpha, skin=0.5)
    t = ew.compute_forces(s)
    e, e_mag, f, f_mag = direct(pos, box, q, mol, rc, alpha, md.coulomb_prefactor())
    assert t["reciprocal"] == 0.0 and abs(t["real"] - e) <= 1e-12 * (1 + e_mag)
    # the intramolecular correction shares the forces: taken off through its own pairs
    intra = np.zeros((n, 3))
    mag = np.zeros((n, 3))
    for i in range(n):
        for j in np.flatnonzero(mol == mol[i]):
            if j != i:
                d = pos[i] - pos[j]
                d -= box * np.round(d / box)
                r = np.linalg.norm(d)
                w = md.coulomb_prefactor() * q[i] * q[j] * (
                    2 * alpha / math.sqrt(math.pi) * math.exp(-(alpha * r) ** 2) - math.erf(alpha * r) / r)
                intra[i] += w / r ** 2 * d
                mag[i] += np.abs(w / r ** 2 * d) + abs(md.coulomb_prefactor() * q[i] * q[j] / r ** 2)
    assert np.all(np.abs(s.forces - f - intra) <= 1e-12 * (1 + f_mag + mag))
