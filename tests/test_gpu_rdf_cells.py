"""The cell pass of the radial distribution function against the oracle's all-pairs
histogram, exactly: crowded cells (more atoms than a staged tile), empty ones, distances on
bin edges, oblong boxes, unwrapped positions, many bins."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,box,rmax,bins", [
    (2, (9.0, 9.0, 9.0), 3.0, 7),
    (33, (9.5, 12.0, 15.0), 3.0, 100),
    (1500, (9.1, 9.2, 9.3), 3.0, 200),       # 27 cells of 55 atoms
    (4200, (9.0, 9.0, 27.0), 3.0, 50),
    (3000, (60.0, 60.0, 60.0), 2.0, 9000),   # mostly empty cells; bins past the shared histogram
])
def test_random_atoms(md, n, box, rmax, bins):
    rng = np.random.default_rng(n)
    box = np.array(box)
    pos = (rng.random((n, 3)) - 0.5) * box
    crowd = n // 6  # a sixth of the atoms in one cell: more than one tile for the larger cases
    pos[:crowd] = 0.3 * rng.random((crowd, 3)) * rmax
    s = md.System.from_arrays(pos, box)
    rdf = md.Rdf(rmax, bins)
    rdf.accumulate(s)
    hist, _ = O.rdf([pos], box, rmax, bins)
    assert np.array_equal(rdf.histogram(), hist)


def test_distances_on_bin_edges(md):
    """A lattice of spacing 0.25 with bins of 0.125: every axial distance is an edge."""
    k = np.arange(-16, 16) * 0.25
    pos = np.stack(np.meshgrid(k, k[:6], k[:6], indexing="ij"), -1).reshape(-1, 3)
    box = np.array([8.0, 9.0, 9.0])
    rdf = md.Rdf(2.0, 16)
    rdf.accumulate(md.System.from_arrays(pos, box))
    hist, _ = O.rdf([pos], box, 2.0, 16)
    assert np.array_equal(rdf.histogram(), hist)
