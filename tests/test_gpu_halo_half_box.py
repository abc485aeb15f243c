"""A cutoff of more than half the box over a list with FP64 halo tiles: a listed pair that has
drifted to exactly half a box length keeps the sign that the gathered pass gives its force."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_pair_at_half_the_box(md, axis):
    box = np.full(3, 16.0)
    pos, vel = np.zeros((2, 3)), np.zeros((2, 3))
    pos[:, axis], vel[1, axis] = [-4.0, -3.0], 7.0
    pos[1, (axis + 1) % 3] = 0.5
    out = []
    for tiles in (False, True):
        s = md.System.from_arrays(pos, box, vel=np.zeros((2, 3)), mass=np.ones(2))
        v = md.VerletList(box, 2.5, 0.3)
        v.build(s)
        v.set_halo(tiles)
        s.velocities = vel
        md.VelocityVerlet(1.0).step(s, lambda sys: None)  # 8 apart, the list as it was
        ev = md.LennardJones(1.0, 1.0, 9.0).compute_forces(s, v)
        out.append((ev, s.forces))
    assert np.all(out[0][1][:, axis] != 0.0)
    assert out[1][0] == out[0][0] and np.array_equal(out[1][1], out[0][1])
