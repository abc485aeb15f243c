"""The FP64 batched force pass: every replica's trajectory equals its solo run bit for bit, in
each thread shape, truncated and shifted; and the shifted potential keeps the truncated one's
pace (it spilled to 1.26 times its time)."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def replica(md, reps, rho, trunc, shape=(0, 0), seed=1):
    a = (4.0 / rho) ** (1.0 / 3.0)
    cell = np.stack(np.meshgrid(*[np.arange(reps)] * 3, indexing="ij"), -1).reshape(-1, 3)
    basis = np.array([[0, 0, 0], [.5, .5, 0], [.5, 0, .5], [0, .5, .5]])
    rng = np.random.default_rng(seed)
    box = np.full(3, reps * a)
    pos = ((cell[:, None, :] + basis).reshape(-1, 3) + 0.25) * a - 0.5 * box
    pos += rng.uniform(-0.1, 0.1, pos.shape)
    ctx = md.Context(0)
    s = md.System.from_arrays(pos, box, vel=rng.normal(size=pos.shape), mass=np.ones(len(pos)), ctx=ctx)
    lj = md.LennardJones(1.0, 1.0, 2.5, trunc)
    lj.set_launch(*shape)
    v = md.VerletList(box, 2.5, 0.3, ctx=ctx)
    v.build(s)
    lj.compute_forces(s, v)
    return md.VelocityVerlet(0.003), s, v, lj


@pytest.mark.parametrize("trunc", [0, 1])
@pytest.mark.parametrize("tpa", [1, 2, 4, 8])
def test_replicas_equal_their_solo_runs(md, tpa, trunc):
    args = [(3, 0.8442), (6, 0.1), (9, 0.8442), (13, 0.5)]
    solo = [replica(md, r, rho, trunc, (tpa, 2), k) for k, (r, rho) in enumerate(args)]
    both = [replica(md, r, rho, trunc, (tpa, 2), k) for k, (r, rho) in enumerate(args)]
    b = md.Batch()
    for r in both:
        b.add(*r)
    rows = b.run(25, thermo=True)
    for k, (it, s, v, lj) in enumerate(solo):
        assert np.array_equal(it.run(s, v, lj, 25, thermo=True), rows[k])
        assert np.array_equal(s.positions, both[k][1].positions)
        assert np.array_equal(s.velocities, both[k][1].velocities)


def test_pace(md):
    """Eight liquids of 32,000 and 70,304 atoms: shifted within 1.2 times truncated (1.14
    measured), the two in turn."""
    runs, times = [], ([], [])
    for trunc in (0, 1):
        keep = [replica(md, 20 + 6 * (k % 2), 0.8442, trunc) for k in range(8)]
        b = md.Batch()
        for r in keep:
            b.add(*r)
        b.run(20)
        runs.append((b, keep))
    for _ in range(9):
        for (b, _), t in zip(runs, times):
            a = time.perf_counter()
            b.run(40)
            t.append(time.perf_counter() - a)
    assert min(times[1]) < 1.2 * min(times[0])
