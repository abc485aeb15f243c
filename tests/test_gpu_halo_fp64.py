"""FP64 forces over halo tiles: bit for bit those of the gathered kernel -- forces, energy,
virial and a fused run's trajectory -- whether every tile is staged (a liquid), none is (a
gas whose blocks span too many cells) or some are (a half-filled box), for tile counts with
a remainder, both truncations and oblong boxes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def box_of_atoms(reps, rho, seed, fill=1.0, missing=0):
    rng = np.random.default_rng(seed)
    a = (4.0 / rho) ** (1.0 / 3.0)
    cell = np.stack(np.meshgrid(*[np.arange(k) for k in reps], indexing="ij"), -1).reshape(-1, 3)
    basis = np.array([[0, 0, 0], [.5, .5, 0], [.5, 0, .5], [0, .5, .5]])
    box = a * np.array(reps, float)
    pos = ((cell[:, None, :] + basis).reshape(-1, 3) + 0.25) * a - 0.5 * box
    pos = pos[pos[:, 2] < (fill - 0.5) * box[2]]
    pos = rng.permutation(pos)[missing:] + rng.uniform(-0.1, 0.1, (len(pos) - missing, 3))
    pos -= box * np.floor(pos / box + 0.5)
    return pos, rng.normal(size=pos.shape), box


def wrapped_system(md, pos, box):
    """The system after a drift of zero velocities: an integrator wrote (and wrapped) its
    positions, which tiles need; positions a caller set are gathered."""
    s = md.System.from_arrays(pos, box, mass=np.ones(len(pos)))
    md.VelocityVerlet(0.001).step(s, lambda sys: None)
    assert np.array_equal(s.positions, pos)
    return s


def test_unwrapped_positions_gather(md):
    """Positions set a box length away give the same forces, tiles on."""
    pos, _, box = box_of_atoms((8, 8, 8), 0.8442, 6)
    out = []
    for shift in (0.0, 1.0):
        p = pos.copy()
        p[::3] += shift * box
        s = md.System.from_arrays(p, box, mass=np.ones(len(pos)))
        v = md.VerletList(box, 2.5, 0.3)
        v.build(s)
        v.set_halo(True)
        md.LennardJones(1.0, 1.0, 2.5).compute_forces(s, v)
        out.append(s.forces)
    # a coordinate moved by a box length is rounded once more: 2 eps L against a slope of
    # the force below 2e3 in this lattice
    assert np.abs(out[1] - out[0]).max() < 80 * 2e3 * 2.3e-16 * box.max()


@pytest.mark.parametrize("trunc", [0, 1])
@pytest.mark.parametrize("reps,rho,fill,missing,staged", [
    ((11, 11, 11), 0.8442, 1.0, 0, "all"),
    ((9, 12, 14), 0.8442, 1.0, 77, "all"),
    ((12, 12, 12), 0.02, 1.0, 1, "none"),
    ((12, 12, 16), 0.8, 0.5, 5, "some"),
])
def test_forces_bit_identical(md, reps, rho, fill, missing, staged, trunc):
    pos, _, box = box_of_atoms(reps, rho, 3, fill, missing)
    s = wrapped_system(md, pos, box)
    v = md.VerletList(box, 2.5, 0.3)
    v.build(s)
    lj = md.LennardJones(1.0, 1.0, 2.5, trunc)
    lj.set_launch(2, 1)  # the plain two-thread walk, whatever the size
    e0, w0 = lj.compute_forces(s, v)
    f0 = s.forces
    v.set_halo(True)
    got, tiles = v.halo_tiles()
    assert tiles > 0 and {"all": got == tiles, "none": got == 0, "some": 0 < got < tiles}[staged]
    e1, w1 = lj.compute_forces(s, v)
    assert np.array_equal(s.forces, f0)
    assert e1 == e0 and w1 == w0


def test_close_pairs_take_the_ieee_division(md):
    """A pair far closer than the fast quotients' range, staged."""
    pos, _, box = box_of_atoms((8, 8, 8), 0.8442, 4)
    pos[0], pos[1] = [0.0, 0.0, 0.0], [3e-17, 0.0, 0.0]
    s = wrapped_system(md, pos, box)
    v = md.VerletList(box, 2.5, 0.3)
    v.build(s)
    lj = md.LennardJones(1.0, 1.0, 2.5)
    lj.compute_forces(s, v)
    f0 = s.forces
    v.set_halo(True)
    lj.compute_forces(s, v)
    assert np.array_equal(s.forces, f0)


def test_fused_run_bit_identical(md):
    """197,000 atoms run over tiles by default; the trajectory and thermo rows through
    several rebuilds equal the gathered run's."""
    pos, vel, box = box_of_atoms((37, 37, 36), 0.8442, 5, missing=112)
    out = []
    for halo in (True, False):
        s = md.System.from_arrays(pos, box, vel=vel, mass=np.ones(len(pos)))
        lj = md.LennardJones(1.0, 1.0, 2.5)
        lj.set_halo(halo)
        v = md.VerletList(box, 2.5, 0.3)
        v.build(s)
        lj.compute_forces(s, v)
        rows = md.VelocityVerlet(0.005).run(s, v, lj, 25, thermo=True)
        assert (v.halo_tiles()[0] > 0) == halo and v.rebuild_count() > 2
        out.append((rows, s.positions, s.velocities))
    assert all(np.array_equal(a, b) for a, b in zip(*out))
