"""Runs of small systems from several threads overlap: each thread waits for its own steps without keeping
the others from launching. Four systems together must take less than 2.5 times as long as one (they
fill a tenth of the GPU each; runs that wait for one another take four times as long)."""
import threading
import time

import numpy as np
import pytest

from helpers import jittered_lattice

pytestmark = pytest.mark.gpu


def voronoi():
    import cellgpu_b200 as cg

    pos, box = jittered_lattice(20, 15, 0.2, 1)
    b = cg.VoronoiBatch([len(pos)], [box])
    b.set_positions(pos)
    b.set_preferences(np.tile([1.0, 3.8], (len(pos), 1)))
    b.set_motility(np.tile([0.05, 1.0], (len(pos), 1)))
    b.set_directors(np.zeros(len(pos)))
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


@pytest.mark.parametrize("make,run", [(voronoi, lambda b: b.spp_run(2000)), (vertex, lambda b: b.brownian_run(2000))])
def test_four_threads_overlap(cglib, make, run):
    systems = [make() for _ in range(4)]

    def together(batch):
        threads = [threading.Thread(target=run, args=(b,)) for b in batch]
        t0 = time.perf_counter()
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        return time.perf_counter() - t0

    for b in systems:
        run(b)
    one = min(together(systems[:1]) for _ in range(5))
    four = min(together(systems) for _ in range(5))
    assert four < 2.5 * one
