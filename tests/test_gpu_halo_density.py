"""FP64 fused runs take halo tiles only where nearly all of them would be staged: not in a gas,
whose blocks of atoms span too many cells, and not with a long cutoff, whose cells overfill a
tile; a caller's own set_halo() decides over that rule, and the trajectory is the same."""
import numpy as np
import pytest

from test_gpu_halo_fp64 import box_of_atoms

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("reps,rho,rc,tiles", [
    ((37, 37, 37), 0.3, 2.5, False),     # 202,612 atoms, 6.9 a cell
    ((37, 37, 37), 0.8442, 4.0, False),  # 74 a cell
    ((37, 37, 37), 0.8442, 2.5, True),
    ((36, 36, 36), 0.8442, 2.5, False),  # 186,624 atoms
])
def test_rule(md, reps, rho, rc, tiles):
    pos, vel, box = box_of_atoms(reps, rho, 5)
    s = md.System.from_arrays(pos, box, vel=vel, mass=np.ones(len(pos)))
    lj = md.LennardJones(1.0, 1.0, rc)
    v = md.VerletList(box, rc, 0.3)
    v.build(s)
    lj.compute_forces(s, v)
    md.VelocityVerlet(0.002).run(s, v, lj, 3)
    staged, total = v.halo_tiles()
    assert (total > 0) == tiles
    if tiles:
        assert staged > 0.95 * total


def test_asked_for_tiles_are_used(md):
    """The gas with tiles the caller asked for: the same trajectory, and tiles kept."""
    pos, vel, box = box_of_atoms((37, 37, 37), 0.3, 5)
    out = []
    for asked in (False, True):
        s = md.System.from_arrays(pos, box, vel=vel, mass=np.ones(len(pos)))
        lj = md.LennardJones(1.0, 1.0, 2.5)
        v = md.VerletList(box, 2.5, 0.3)
        v.build(s)
        if asked:
            v.set_halo(True)
        lj.compute_forces(s, v)
        rows = md.VelocityVerlet(0.004).run(s, v, lj, 20, thermo=True)
        assert (v.halo_tiles()[1] > 0) == asked and v.rebuild_count() > 1
        out.append((rows, s.positions, s.velocities))
    assert all(np.array_equal(x, y) for x, y in zip(*out))
