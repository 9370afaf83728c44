"""Systems that run at the same time, from several threads or one, share the GPU: each thread waits for its
own steps without keeping the others from launching, and launches that would fill the GPU take their
share of it. Bounds on times are halfway between runs that overlap and runs that take turns (four times
as long as one)."""
import threading
import time

import numpy as np
import pytest

from helpers import jittered_lattice

pytestmark = pytest.mark.gpu


def voronoi(nx=20, ny=15, det=False):
    import cellgpu_b200 as cg

    pos, box = jittered_lattice(nx, ny, 0.2, 1)
    b = cg.VoronoiBatch([len(pos)], [box])
    b.set_positions(pos)
    b.set_preferences(np.tile([1.0, 3.8], (len(pos), 1)))
    b.set_motility(np.tile([0.05, 1.0], (len(pos), 1)))
    b.set_directors(np.zeros(len(pos)))
    b.set_deterministic(det)
    b.triangulate()
    return b


def vertex():
    import cellgpu_b200 as cg

    pos, box = jittered_lattice(20, 15, 0.2, 1)
    b = cg.VertexBatch([len(pos)], [box])
    b.from_cells(pos)
    b.set_preferences(np.tile([1.0, 3.8], (len(pos), 1)))
    b.set_t1_threshold(0.04)
    return b


def together(batch, run):
    threads = [threading.Thread(target=run, args=(b,)) for b in batch]
    t0 = time.perf_counter()
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return time.perf_counter() - t0


@pytest.mark.parametrize("make,run", [(voronoi, lambda b: b.spp_run(2000)), (vertex, lambda b: b.brownian_run(2000))])
def test_four_threads_overlap(cglib, make, run):
    systems = [make() for _ in range(4)]
    for b in systems:
        run(b)
    one = min(together(systems[:1], run) for _ in range(5))
    four = min(together(systems, run) for _ in range(5))
    assert four < 2.5 * one


def test_minimisations_that_fill_the_gpu_share_it(cglib):
    import cellgpu_b200 as cg

    prm = cg.FireParams.defaults(force_cutoff=1e-13, max_iterations=10**6)
    systems = [voronoi(128, 128) for _ in range(4)]
    for b in systems:
        b.fire_begin(prm)
    run = lambda b: b.fire_advance(prm, 1024)
    for b in systems:
        run(b)
    one = min(together(systems[:1], run) for _ in range(3))
    four = min(together(systems, run) for _ in range(3))
    assert four < 3.0 * one


def test_single_steps_of_several_streams_overlap(cglib):
    systems = [voronoi(128, 128) for _ in range(4)]

    def steps(batch):
        t0 = time.perf_counter()
        for _ in range(100):
            for b in batch:
                assert cglib.cg_spp_enqueue(b.handle, 1, 0.01, 1.0) == 0
        for b in batch:
            assert cglib.cg_synchronize(b.handle) == 0
        return time.perf_counter() - t0

    steps(systems)
    one = min(steps(systems[:1]) for _ in range(3))
    four = min(steps(systems) for _ in range(3))
    assert four < 2.5 * one


@pytest.mark.parametrize("nx,ny", [(40, 37), (128, 128), (182, 182)])
def test_shared_launches_change_no_bit(cglib, nx, ny):
    """Deterministic runs beside three others (smaller grids) end in the bits of a run alone, single steps
    through the graph too."""
    alone = voronoi(nx, ny, det=True)
    alone.spp_run(300)
    alone.spp_run(1)
    systems = [voronoi(nx, ny, det=True) for _ in range(4)]

    def run(b):
        for _ in range(3):
            b.spp_run(100)

    together(systems, run)
    for b in systems:
        assert cglib.cg_spp_enqueue(b.handle, 1, 0.01, 1.0) == 0
    for b in systems:
        assert cglib.cg_synchronize(b.handle) == 0
        assert np.array_equal(b.positions(), alone.positions())
        assert np.array_equal(b.directors(), alone.directors())
