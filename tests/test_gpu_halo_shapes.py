"""Launch shapes and halo tiles in FP64: forces, energy and virial with tiles on are those of the
gathered pass in the shape the caller asked for, bit for bit, and a fused run builds tiles only
for the shape that reads them; the autotuner's cache keeps such cases apart."""
import numpy as np
import pytest

import moleculardynamics_b200.autotune as T
from test_gpu_halo_fp64 import box_of_atoms, wrapped_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1), (2, 4), (4, 2), (8, 1), (0, 0)])
def test_tiles_keep_the_shape(md, shape):
    pos, _, box = box_of_atoms((11, 11, 11), 0.8442, 3)
    s = wrapped_system(md, pos, box)
    v = md.VerletList(box, 2.5, 0.3)
    v.build(s)
    lj = md.LennardJones(1.0, 1.0, 2.5)
    lj.set_launch(*shape)
    gathered = lj.compute_forces(s, v), s.forces
    v.set_halo(True)
    tiled = lj.compute_forces(s, v), s.forces
    assert tiled[0] == gathered[0] and np.array_equal(tiled[1], gathered[1])


def test_run_in_another_shape_builds_no_tiles(md):
    pos, vel, box = box_of_atoms((37, 37, 37), 0.8442, 5)
    for shape, tiles in (((4, 2), False), ((2, 2), True)):
        s = md.System.from_arrays(pos, box, vel=vel, mass=np.ones(len(pos)))
        lj = md.LennardJones(1.0, 1.0, 2.5)
        lj.set_launch(*shape)
        v = md.VerletList(box, 2.5, 0.3)
        v.build(s)
        lj.compute_forces(s, v)
        md.VelocityVerlet(0.004).run(s, v, lj, 2)
        assert (v.halo_tiles()[1] > 0) == tiles


def test_cache_keys(md):
    lj = md.LennardJones(1.0, 1.0, 2.5)
    keys = []
    for reps in (13, 14, 21, 22):  # 8,788 and 10,976 atoms; 37,044 and 42,592: 64 and 256 an SM
        pos, _, box = box_of_atoms((reps,) * 3, 0.8442, 2)
        s = md.System.from_arrays(pos, box, mass=np.ones(len(pos)))
        v = md.VerletList(box, 2.5, 0.3)
        v.build(s)
        keys.append(T.problem_key(s.ctx, s, lj, 2.5, 0.3, v))
    v.set_halo(True)
    keys.append(T.problem_key(s.ctx, s, lj, 2.5, 0.3, v))
    assert len(set(keys)) == 5
