"""The shapes of the g(r) cell pass: few cells shared by several blocks, sparse cells with a
thread an atom, a crowd among sparse cells, blocks that walk the cells, each against the
oracle's all-pairs histogram, exactly; coordinates several box lengths away and subsets; and
frames whose time must not depend on the number of cells alone."""
import ctypes as C
import time

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def scattered(n, box, seed, clump=0, width=1.0):
    rng = np.random.default_rng(seed)
    pos = (rng.random((n, 3)) - 0.5) * box
    pos[:clump] = width * rng.random((clump, 3)) + 0.2 * box
    return pos


@pytest.mark.parametrize("n,box,rmax,bins,clump,width", [
    (1100, (9.1, 9.2, 9.3), 3.0, 40, 0, 1.0),       # 27 cells, a slice each: mean just over 4 x 128 / 14
    (4000, (9.1, 9.2, 9.3), 3.0, 300, 0, 1.0),      # 27 cells, four slices
    (4000, (9.1, 9.2, 9.3), 3.0, 300, 1500, 2.9),   # uneven, tiles with a remainder
    (3000, (46.0, 46.0, 46.0), 2.0, 100, 0, 1.0),   # 12,167 sparse cells
    (6000, (46.0, 46.0, 46.0), 2.0, 8192, 900, 1.9),  # a crowd of several slices among them
    (6000, (46.0, 46.0, 46.0), 2.0, 9000, 900, 6.0),  # spread over cells; no shared histogram
    (5000, (20.0, 20.0, 40.0), 2.0, 2000, 0, 1.0),  # 2,000 cells walked
    (5000, (20.0, 20.0, 40.0), 2.0, 2000, 300, 1.5),
])
def test_shapes(md, n, box, rmax, bins, clump, width):
    box = np.array(box)
    pos = scattered(n, box, n + bins, clump, width)
    rdf = md.Rdf(rmax, bins)
    rdf.accumulate(md.System.from_arrays(pos, box))
    hist, _ = O.rdf([pos], box, rmax, bins)
    assert np.array_equal(rdf.histogram(), hist)


@pytest.mark.parametrize("box,rmax", [((9.1, 9.2, 9.3), 3.0), ((46.0, 46.0, 46.0), 2.0)])
@pytest.mark.parametrize("first,stride", [(0, 1), (1, 3)])
def test_unwrapped_and_subsets(md, box, rmax, first, stride):
    rng = np.random.default_rng(first + 5)
    box = np.array(box)
    pos = scattered(3000, box, 8, 400, 1.8)
    moved = rng.random(len(pos)) < 0.4
    pos[moved] += rng.integers(-2, 3, (moved.sum(), 3)) * box
    rdf = md.Rdf(rmax, 100)
    rdf.accumulate(md.System.from_arrays(pos, box), first, stride)
    hist, _ = O.rdf([pos[first::stride]], box, rmax, 100)
    assert np.array_equal(rdf.histogram(), hist)


@pytest.mark.parametrize("rmax,bins", [(2.7, 60), (3.5, 3000), (19.0, 100)])
def test_frames_in_a_captured_block(md, rmax, bins):
    """A droplet of water: the frames that md_water_rdf_run's graph takes (sparse cells, walked
    cells, 27 cells) are those of separate calls on the same trajectory."""
    half = np.radians(0.5 * 109.47)
    body = np.array([[0, 0, 0], [np.sin(half), 0, np.cos(half)], [-np.sin(half), 0, np.cos(half)]])
    grid = np.stack(np.meshgrid(*[np.arange(7)] * 3, indexing="ij"), -1).reshape(-1, 3) - 3.0
    rng = np.random.default_rng(5)
    turn = np.linalg.qr(rng.normal(size=(len(grid), 3, 3)))[0]
    pos = (3.1 * grid[:, None] + np.einsum("mij,kj->mki", turn, body)).reshape(-1, 3)
    m = len(grid)
    vel = np.repeat(3.0 * rng.normal(size=(m, 3)), 3, axis=0)
    dof, hist = md.RigidWater.degrees_of_freedom(m, True), []
    for fused in (True, False):
        s = md.System.from_arrays(pos, np.full(3, 60.0), vel=vel, mass=np.tile([15.9994, 1.008, 1.008], m),
                                  charge=np.tile([-0.8476, 0.4238, 0.4238], m), mol=np.arange(3 * m) // 3)
        rigid = md.RigidWater(1.0, 109.47, settle=True)
        rigid.constrain_velocities(s)
        it = md.ConstrainedVelocityVerlet(md.units.femtoseconds(1.0), rigid)
        ff, rdf = md.SpceForceField(), md.Rdf(rmax, bins)
        if fused:
            t = C.c_double()
            md._check(md.lib().md_water_rdf_run(it.handle, s.handle, ff.handle, rdf.handle, 298.0, dof,
                                                20, 10, 40, 5, C.byref(t)))
        else:
            for _ in range(2):
                it.run(s, ff, 10)
                s.rescale_temperature(dof, 298.0)
                rigid.constrain_velocities(s)
            for _ in range(8):
                it.run(s, ff, 5)
                rdf.accumulate(s, 0, 3)
        hist.append(rdf.histogram())
    assert hist[0].sum() > 0 and np.array_equal(hist[0], hist[1])


def frame_time(md, pos, box, rmax, bins):
    s = md.System.from_arrays(pos, box)
    rdf = md.Rdf(rmax, bins)
    times = []
    for _ in range(6):
        md.default_context().synchronize()
        t = time.perf_counter()
        rdf.accumulate(s)
        md.default_context().synchronize()
        times.append(time.perf_counter() - t)
    return min(times[1:])


def test_few_cells_keep_the_gpu_busy(md):
    """27 cells hold every pair; the pass over them takes at most three times the all-pairs
    pass of the same atoms (551 and 420 us measured; one block a cell took 3,240)."""
    box = np.full(3, 23.5)
    pos = scattered(10976, box, 3)
    assert frame_time(md, pos, box, 7.8, 200) < 3 * frame_time(md, pos, box, 11.7, 200)


def test_sparse_cells_cost_no_block_each(md):
    """Fewer pairs in more cells: rMax 1.5 with 8,000 bins takes no longer than rMax 4 (107 and
    190 us measured; a block a cell with a histogram each took 1,830 and 350)."""
    box = np.full(3, 102.6)
    pos = scattered(108000, box, 4)
    assert frame_time(md, pos, box, 1.5, 8000) < 1.5 * frame_time(md, pos, box, 4.0, 8000)
