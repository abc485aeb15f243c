"""Systems on either side of the block sizes of the position update: a fused run, whose update
also checks the displacements, equals single steps with the list's own check bit for bit and
rebuilds as often."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["vv", "baoab"])
@pytest.mark.parametrize("cells", [3, 10, 11, 21, 22])
def test_fused_run_equals_single_steps(md, cells, kind):
    st = md.fcc_lattice(cells, 0.7, 2.0, 9)
    keep = len(st["pos"]) - 3  # a ragged last block
    out = []
    for fused in (True, False):
        s = md.System.from_arrays(st["pos"][:keep], st["box"], vel=st["vel"][:keep],
                                  mass=st["mass"][:keep])
        lj = md.LennardJones(1.0, 1.0, 2.5)
        v = md.VerletList(st["box"], 2.5, 0.3)
        v.build(s)
        lj.compute_forces(s, v)
        it = md.VelocityVerlet(0.006) if kind == "vv" else md.LangevinBAOAB(0.006, 1.0, 2.0, 3)
        if fused:
            it.run(s, v, lj, 24)
        else:
            for _ in range(24):
                it.step(s, lambda sys: (v.rebuild_if_needed(sys), lj.compute_forces(sys, v)))
        out.append((s.positions, s.velocities, v.rebuild_count()))
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])
    assert out[0][2] == out[1][2] > 1
