"""Fused Langevin runs replay a captured step whose noise counter lives on the device: the
trajectory equals host launches bit for bit over calls of several lengths, through rebuilds,
and the step counter that a later single step continues from is the same."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("cells", [3, 7, 26])  # all-pairs list; cells; halo tiles (mixed)
def test_replay_equals_host_launches(md, cells, mixed):
    st = md.fcc_lattice(cells, 0.8, 1.1, 5)
    prec = md.PRECISION_MIXED if mixed else md.PRECISION_FP64
    out = []
    for graphs in (False, True):
        ctx = md.Context(0)
        ctx.set_graphs(graphs)
        s = md.System.from_arrays(st["pos"], st["box"], vel=st["vel"], mass=st["mass"], ctx=ctx)
        lj = md.LennardJones(1.0, 1.0, 2.5, precision=prec)
        v = md.VerletList(st["box"], 2.5, 0.3, ctx=ctx)
        v.build(s)
        lj.compute_forces(s, v)
        it = md.LangevinBAOAB(0.005, 1.0, 1.1, 77)
        rows = [it.run(s, v, lj, k, thermo=True) for k in (1, 3, 24, 2)]
        it.step(s, lambda sys: (v.rebuild_if_needed(sys), lj.compute_forces(sys, v)))
        rows.append(it.run(s, v, lj, 5, thermo=True))
        assert v.rebuild_count() > 2
        assert (ctx.graph_captures() > 0) == graphs
        out.append((np.concatenate(rows), s.positions, s.velocities))
    assert all(np.array_equal(a, b) for a, b in zip(*out))


def test_replayed_noise_still_steps_from_the_host(md):
    st = md.fcc_lattice(3, 0.8, 1.1, 6)
    xi = np.random.default_rng(1).normal(size=3 * len(st["pos"]) * 4)
    out = []
    for steps in ((4,), (1, 3)):
        s = md.System.from_arrays(st["pos"], st["box"], vel=st["vel"], mass=st["mass"])
        lj = md.LennardJones(1.0, 1.0, 2.5)
        v = md.VerletList(st["box"], 2.5, 0.3)
        v.build(s)
        lj.compute_forces(s, v)
        it = md.LangevinBAOAB(0.005, 1.0, 1.1, 77)
        it.set_noise(xi)
        for k in steps:
            it.run(s, v, lj, k)
        out.append(s.positions)
        with pytest.raises(md.InvalidArgument):
            it.run(s, v, lj, 1)  # the noise is used up
    assert np.array_equal(*out)
