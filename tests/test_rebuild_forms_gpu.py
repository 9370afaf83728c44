"""Steps and FIRE iterations that the local repair cannot finish, in every form that runs them: each
halts, the triangulation is rebuilt globally and the run goes on.

SPP: with mu = 0 and v0 dt above a cell's size the positions do not depend on the forces and every cell
leaves its neighbours in each step, so positions must equal the oracle's integration to rounding.
FIRE: two iterations of a time step large enough to tear the tissue. After the first move the positions
agree to rounding, so the second one adds the error of one force evaluation (1e-8 of the force, the
suite's tolerance) times dt^2 = 4 and a margin of 25 for the kicks and the mix."""
import numpy as np
import pytest

from helpers import jittered_lattice

pytestmark = pytest.mark.gpu


def lattices(sizes):
    pts, boxes = zip(*[jittered_lattice(nx, ny, 0.35, 11 + i) for i, (nx, ny) in enumerate(sizes)])
    return list(pts), list(boxes)


# one cluster, a few blocks, a full grid, uneven instances, the thread-per-cell pass, two launches a step
@pytest.mark.parametrize("sizes,det", [([(20, 15)], False), ([(33, 32)], True), ([(96, 100)], False),
                                       ([(20, 15), (40, 41), (25, 24)], False), ([(182, 182)], False),
                                       ([(182, 182)], True)])
def test_spp_steps_rebuild(cglib, oracle, sizes, det):
    import torch
    import cellgpu_b200 as cg

    steps = 4
    pts, boxes = lattices(sizes)
    n = sum(len(p) for p in pts)
    rng = np.random.default_rng(n)
    theta = rng.uniform(0, 2 * np.pi, n)
    mot = np.tile([1.5, 1.0], (n, 1))
    noise = rng.standard_normal((steps, n))
    b = cg.VoronoiBatch([len(p) for p in pts], boxes)
    b.set_positions(np.concatenate(pts))
    b.set_directors(theta)
    b.set_preferences(np.tile([1.0, 3.8], (n, 1)))
    b.set_motility(mot)
    if det:
        b.set_deterministic(True)
    b.triangulate()
    before = b.counters()["global_rebuilds"]
    b.spp_run(steps, dt=1.0, mu=0.0, noise=torch.tensor(noise, device="cuda:0"))
    assert b.counters()["global_rebuilds"] - before >= steps - 1
    b.enforce_topology()
    got, nn, nbr = b.positions(), *b.topology()
    off = 0
    for p, box in zip(pts, boxes):
        at = slice(off, off + len(p))
        want, th = p.copy(), theta[at].copy()
        for t in range(steps):
            oracle.spp_step(want, box, np.zeros_like(want), th, mot[at], noise[t, at], 1.0, 0.0)
        d = got[at] - want
        d -= np.round(d / np.array(box)) * np.array(box)
        assert np.abs(d).max() < 1e-11
        rows = np.where(nbr[at] >= 0, nbr[at] - off, -1)
        assert oracle.topology_mismatch(got[at], box, nn[at], np.ascontiguousarray(rows, np.int32)) == 0
        off += len(p)


@pytest.mark.parametrize("nx,ny", [(20, 15), (96, 100), (182, 182)])
def test_fire_iterations_rebuild(cglib, oracle, nx, ny):
    import cellgpu_b200 as cg

    (pos,), (box,) = lattices([(nx, ny)])
    n = len(pos)
    pref = np.tile([1.0, 3.8], (n, 1))
    opts = dict(dt=2.0, dt_max=2.0, force_cutoff=1e-12, max_iterations=2)
    b = cg.VoronoiBatch([n], [box])
    b.set_positions(pos)
    b.set_preferences(pref)
    b.triangulate()
    before = b.counters()["global_rebuilds"]
    b.fire_minimize(cg.FireParams.defaults(**opts))
    assert b.counters()["global_rebuilds"] > before
    assert b.fire_state()[0][0] == 2
    nn, nbr = oracle.periodic_delaunay(pos, box, 16)
    want = pos.copy()
    F, _, _ = oracle.fire_voronoi(want, box, nn, nbr, pref, oracle.FireParams.defaults(**opts))
    d = b.positions() - want
    d -= np.round(d / np.array(box)) * np.array(box)
    assert np.abs(d).max() < 1e-6 * np.abs(F).max()
    gnn, gnbr = b.topology()
    assert oracle.topology_mismatch(b.positions(), box, gnn, gnbr) == 0


@pytest.mark.parametrize("nx,ny", [(33, 32), (96, 100)])
def test_fire_with_more_rebuilds_than_chunks(cglib, nx, ny):
    """A time step so long that nearly every iteration needs a rebuild: 160 iterations, each of which may end
    its launch, run through (10 chunks of 16; the oracle's run of the same parameters stays finite)."""
    import cellgpu_b200 as cg

    (pos,), (box,) = lattices([(nx, ny)])
    n = len(pos)
    b = cg.VoronoiBatch([n], [box])
    b.set_positions(pos)
    b.set_preferences(np.tile([1.0, 3.8], (n, 1)))
    b.triangulate()
    before = b.counters()["global_rebuilds"]
    b.fire_minimize(cg.FireParams.defaults(dt=2.0, dt_max=2.0, dt_min=2.0, force_cutoff=1e-12, max_iterations=160))
    assert b.counters()["global_rebuilds"] - before > 160 // 16 + 64
    assert b.fire_state()[0][0] == 160
    assert np.isfinite(b.positions()).all()
