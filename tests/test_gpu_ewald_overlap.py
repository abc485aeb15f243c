"""Two overlapping oxygens in FP32 real-space terms: infinite forces and energy where
(sigma/r)^12 leaves FP32's range, as divisions give them and never NaN, and the FP64 forces
above that.

Tolerance above it: r^2 is rounded to FP32 (6e-8) and enters to the seventh power, and the
terms have about ten more FP32 roundings: 7 x 6e-8 + 10 x 6e-8, doubled."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BODY = np.array([[0.0, 0.0, 0.0], [0.3, 0.95, 0.0], [0.3, -0.95, 0.1]])


def forces(md, dist, precision):
    """27 waters on a lattice, the second one's oxygen `dist` from the first one's."""
    grid = np.stack(np.meshgrid(*[np.arange(3)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = ((grid[:, None] - 1.0) * 3.5 + BODY).reshape(-1, 3)
    pos[3:6] += pos[0] + dist / np.sqrt(3.0) - pos[3]
    pos[4:6, 2] += 1.0  # its hydrogens away from the first one's
    m = len(grid)
    s = md.System.from_arrays(pos, [10.5] * 3, mass=np.tile([16.0, 1.0, 1.0], m),
                              charge=np.tile([-0.8476, 0.4238, 0.4238], m), mol=np.arange(3 * m) // 3)
    ff = md.SpceForceField(cutoff=5.0, kmax=3)
    ff.set_precision(precision)
    return ff.compute_forces(s), s.forces


@pytest.mark.parametrize("dist", [1e-3, 3e-3])
def test_beyond_fp32(md, dist):
    e, f = forces(md, dist, md.PRECISION_MIXED)
    assert e == np.inf
    assert np.all(f[0] == -np.inf) and np.all(f[3] == np.inf)


@pytest.mark.parametrize("dist", [0.009, 0.0099, 0.011, 0.012, 0.0125, 0.05, 1.0])
def test_within_fp32(md, dist):
    """On either side of the rule that chooses between the division and the quotients."""
    e, f = forces(md, dist, md.PRECISION_MIXED)
    e64, f64 = forces(md, dist, md.PRECISION_FP64)
    assert abs(e - e64) <= 2.1e-6 * abs(e64)
    assert np.abs(f - f64)[[0, 3]].max() <= 2.1e-6 * np.abs(f64).max()
