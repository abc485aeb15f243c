"""The FP64 pair arithmetic and the launch shapes of the gathered force kernel.

Isolated pairs: every atom has at most one partner, so its force is one pair term and has
to equal the oracle's bit for bit (the kernel's shared-reciprocal quotients are correctly
rounded), from separations far below the atoms' size, where the kernel divides in IEEE
arithmetic, to the cutoff.  Small systems: their own launch shape against the batched one,
bit for bit."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("trunc", [0, 1])
@pytest.mark.parametrize("source", ["verlet", "cells", "brute"])
def test_isolated_pairs_bit_exact(md, source, trunc):
    rng = np.random.default_rng(11 + trunc)
    side, gap = 11, 7.0
    box = np.full(3, side * gap)
    cell = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)
    a = (cell - side // 2) * gap + rng.uniform(-0.5, 0.5, (len(cell), 3))
    d = rng.normal(size=a.shape)
    d *= (rng.uniform(0.7, 2.6, len(a)) / np.linalg.norm(d, axis=1))[:, None]
    b = a + d
    mid = len(a) // 2  # the cell at the origin: r far below sigma is representable
    a[mid], b[mid] = 0.0, [3e-17, 0.0, 0.0]
    b[mid + 1] = a[mid + 1] + [1e-3, 0, 0]
    pos = np.stack([a, b], 1).reshape(-1, 3)
    pos -= box * np.floor(pos / box + 0.5)
    s = md.System.from_arrays(pos, box)
    lj = md.LennardJones(1.0, 1.0, 2.5, trunc)
    src = {"verlet": lambda: md.VerletList(box, 2.5, 0.3), "cells": lambda: md.CellList(box, 2.5),
           "brute": lambda: None}[source]()
    if src is not None:
        src.build(s)
    lj.compute_forces(s, src)
    f_ref, _, _ = O.lj_compute(pos, box, rc=2.5, trunc=trunc)
    assert np.array_equal(s.forces, f_ref)


@pytest.mark.parametrize("trunc", [0, 1])
@pytest.mark.parametrize("mixed,cubic", [(False, True), (True, True), (True, False)])
def test_small_systems_equal_their_batch(md, mixed, cubic, trunc):
    """A small FP64 system's own pass takes sixteen lanes an atom, a batch's two; sums, order
    and reduction tree are the same, so forces, energies and kinetic energies are equal bit
    for bit (mixed: two lanes both times).  Sizes around a block of 16 atoms, a warp and a block of the two-thread pass."""
    rng = np.random.default_rng(5)
    a = (4.0 / 0.8) ** (1.0 / 3.0)
    reps = np.array([8, 8, 8] if cubic else [8, 9, 10])
    cell = np.stack(np.meshgrid(*[np.arange(k) for k in reps], indexing="ij"), -1).reshape(-1, 3)
    basis = np.array([[0, 0, 0], [.5, .5, 0], [.5, 0, .5], [0, .5, .5]])
    box = a * reps
    full = ((cell[:, None, :] + basis).reshape(-1, 3) + 0.25) * a - 0.5 * box
    full += rng.uniform(-0.1, 0.1, full.shape)
    vel = rng.normal(size=full.shape)
    prec = md.PRECISION_MIXED if mixed else md.PRECISION_FP64

    def make(n, ctx):
        s = md.System.from_arrays(full[:n], box, vel=vel[:n], mass=np.ones(n), ctx=ctx)
        lj = md.LennardJones(1.0, 1.0, 2.5, trunc, precision=prec)
        v = md.VerletList(box, 2.5, 0.3, ctx=ctx)
        v.build(s)
        return (md.VelocityVerlet(0.004), s, v, lj), lj.compute_forces(s, v), s.forces

    sizes = [1, 15, 16, 17, 33, 127, 129, 1000, 2048]
    batch, parts = md.Batch(), []
    for n in sizes:
        parts.append(make(n, md.Context(0))[0])
        batch.add(*parts[-1])
    rows = batch.run(12, thermo=True)
    for k, n in enumerate(sizes):
        (it, s, v, lj), (e, w), f = make(n, md.Context(0))
        if not mixed:
            f_ref, e_ref, w_ref = O.lj_compute(full[:n], box, rc=2.5, trunc=trunc)
            assert np.all(np.abs(f - f_ref) <= 1e-12 * (1 + np.abs(f_ref))), n
            assert abs(e - e_ref) <= 1e-12 * (1 + abs(e_ref)) and abs(w - w_ref) <= 1e-12 * (1 + abs(w_ref))
        assert np.array_equal(it.run(s, v, lj, 12, thermo=True), rows[k]), n
        assert np.array_equal(parts[k][1].positions, s.positions), n
        assert np.array_equal(parts[k][1].velocities, s.velocities), n


@pytest.mark.parametrize("trunc", [0, 1])
def test_middle_systems_equal_their_batch(md, trunc):
    """From 64 to 256 atoms per SM four lanes take an atom, again with the two-lane sums:
    10,976 atoms (a part of the last block), 23,328 and, back at two lanes, 39,303."""
    def make(cells, missing, ctx):
        st = md.fcc_lattice(cells, 0.75, 1.3, cells)
        keep = slice(missing, None)
        s = md.System.from_arrays(st["pos"][keep], st["box"], vel=st["vel"][keep],
                                  mass=st["mass"][keep], ctx=ctx)
        lj = md.LennardJones(1.0, 1.0, 2.5, trunc)
        v = md.VerletList(st["box"], 2.5, 0.3, ctx=ctx)
        v.build(s)
        lj.compute_forces(s, v)
        return md.NoseHooverChain(0.005, 1.3, 0.5, 3, 3 * s.n - 3), s, v, lj

    sizes = [(14, 0), (14, 41), (18, 0), (22, 3289)]
    batch = md.Batch()
    parts = [make(c, m, md.Context(0)) for c, m in sizes]
    for p in parts:
        batch.add(*p)
    rows = batch.run(15, thermo=True)
    for k, (c, m) in enumerate(sizes):
        it, s, v, lj = make(c, m, md.Context(0))
        assert np.array_equal(it.run(s, v, lj, 15, thermo=True), rows[k]), k
        assert np.array_equal(parts[k][1].positions, s.positions), k
        assert np.array_equal(parts[k][1].velocities, s.velocities), k
