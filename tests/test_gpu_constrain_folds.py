"""SHAKE and RATTLE of molecules that straddle the box's edges, at ordinary masses and at
masses outside the range of the shared-reciprocal quotients (then IEEE divisions): every
bit and the sweep count as the oracle's."""
import numpy as np
import pytest

import oracle as O
from test_gpu_constrain import SPCE, constraint, thermal_velocities, water

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mass_exponent", [0, -120, -420])
def test_constraints_across_the_edges(md, mass_exponent):
    rw, orw = constraint(md)
    src = water(md)
    thermal_velocities(md, src, 298.0, 11)
    box = SPCE["box1"]
    centre = 0.5 * box
    ref = src.positions
    ref = ref - np.repeat(ref[0::3], 3, axis=0)  # every oxygen at a corner of the box
    ref = ref + centre * (np.arange(src.n) // 3 % 2)[:, None]  # or, every other, mid-box
    ref = ref - box * np.floor(ref / box)
    mass = np.ldexp(src.masses, mass_exponent)
    i = np.arange(src.n)
    sh = 0.01 * (i % 7) - 0.03
    disp = ref + np.stack([sh, -0.5 * sh, 0.25 * sh], 1)
    s = md.System.from_arrays(disp, box, vel=src.velocities, mass=mass)
    it = rw.constrain_positions(s, ref)
    want, oit = O.shake(orw, disp, ref, mass, box)
    assert np.array_equal(s.positions, want)
    assert it == oit and it > 1
    it = rw.constrain_velocities(s)
    want, oit = O.rattle(orw, s.positions, src.velocities, mass, box)
    assert np.array_equal(s.velocities, want)
    assert it == oit and it > 1
