"""Halo tiles whose atoms span few cells, many, and too many: forces over the tiles equal the
gathered ones bit for bit, and the tiles are staged where they can be."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rho,some", [(0.8442, True), (0.62, True), (0.45, True), (0.2, False)])
def test_tiles_equal_gathers(md, rho, some):
    st = md.fcc_lattice(9, rho, 1.0, 4)
    rng = np.random.default_rng(8)
    box = st["box"]
    pos = np.mod(st["pos"] + rng.normal(0.0, 0.1, st["pos"].shape), box)
    out = []
    for halo in (True, False):
        s = md.System.from_arrays(pos, box, mass=st["mass"])
        lj = md.LennardJones(1.0, 1.0, 2.5, precision=md.PRECISION_MIXED)
        v = md.VerletList(box, 2.5, 0.3)
        v.build(s)
        v.set_halo(halo)
        staged, tiles = v.halo_tiles()
        assert (staged > tiles // 2) == (halo and some)
        e, w = lj.compute_forces(s, v)
        out.append((e, w, s.forces))
    assert out[0][:2] == out[1][:2] and np.array_equal(out[0][2], out[1][2])
