"""The list builds of sparse cells and of systems too small to fill the GPU: the listed pairs
(exact test at export) equal the oracle's for occupancies around each build's groups of atoms,
windows of candidates and empty cells, and a clump far above the mean."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def gas(n, box, seed, clump=0, width=1.0):
    rng = np.random.default_rng(seed)
    pos = rng.uniform(0.0, 1.0, (n, 3)) * box
    if clump:
        pos[:clump] = rng.uniform(0.0, width, (clump, 3)) + 0.3 * box
    return pos


@pytest.mark.parametrize("n,side,cutoff,clump", [
    (1, 12.0, 2.5, 0),         # every cell but one empty
    (2, 12.0, 2.5, 2),
    (33, 12.0, 2.5, 0),
    (700, 22.5, 2.5, 0),       # sparse, 512 cells
    (1500, 22.5, 2.5, 67),     # sparse with a cell above its warps' atoms
    (217, 8.4, 2.5, 0),        # team, 27 cells at the edge of the rule (8.04 a cell)
    (215, 8.4, 2.5, 0),        # just below it: a lane an atom
    (900, 8.4, 2.5, 97),       # team: a cell of more atoms than a block takes at once
    (3000, 9.0, 2.7, 0),       # team: more candidates than one window holds
    (3000, 9.0, 2.7, 300),     # and several passes over several windows
])
def test_build_lists_the_oracles_pairs(md, n, side, cutoff, clump):
    box = np.array([side, 1.01 * side, 0.99 * side + 0.1])
    pos = gas(n, box, n + clump, clump)
    s = md.System.from_arrays(pos, box, mass=np.ones(n))
    v = md.VerletList(box, cutoff, 0.1)
    v.build(s)
    ref = O.verlet_pairs(pos, box, cutoff, 0.1)
    if len(ref):
        ref = ref[np.lexsort((ref[:, 1], ref[:, 0]))]
        assert np.array_equal(v.pairs(), ref)
    else:
        assert len(v.pairs()) == 0
