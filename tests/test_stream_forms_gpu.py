"""Which form single steps of several systems take: systems that share a stream follow one another and step
in one launch each, systems of several streams go through the
step graph (force pass, repair start, drawn normals, integrator, step end), and alone again a system
returns to one launch."""
import numpy as np
import pytest

from helpers import jittered_lattice

pytestmark = pytest.mark.gpu


def voronoi(seed):
    import cellgpu_b200 as cg

    pos, box = jittered_lattice(20, 15, 0.1, seed)
    b = cg.VoronoiBatch([len(pos)], [box])
    b.set_positions(pos)
    b.set_directors(np.zeros(len(pos)))
    b.set_motility(np.tile([0.01, 1.0], (len(pos), 1)))
    b.set_preferences(np.tile([1.0, 3.8], (len(pos), 1)))
    b.triangulate()
    b.spp_run(20)
    return b


def kernels_of_last_step(cglib, systems):
    """Host-enqueued kernels of the second of two rounds of single steps, per system."""
    before = []
    for k in range(2):
        for b in systems:
            assert cglib.cg_spp_enqueue(b.handle, 1, 0.01, 1.0) == 0
    for b in systems:
        assert cglib.cg_synchronize(b.handle) == 0
        before.append(cglib.cg_kernels_launched(b.handle))
    for k in range(2):
        for b in systems:
            assert cglib.cg_spp_enqueue(b.handle, 1, 0.01, 1.0) == 0
    for b in systems:
        assert cglib.cg_synchronize(b.handle) == 0
    return [cglib.cg_kernels_launched(b.handle) - n for b, n in zip(systems, before)]


def test_forms_by_stream(cglib):
    import torch

    systems = [voronoi(i) for i in range(5)]
    stream = torch.cuda.Stream()
    for b in systems:
        assert cglib.cg_set_stream(b.handle, stream.cuda_stream) == 0
    assert kernels_of_last_step(cglib, systems) == [2] * 5
    for b in systems:
        assert cglib.cg_set_stream(b.handle, None) == 0
    n = kernels_of_last_step(cglib, systems)
    # five kernels and two for each repair round by the graph; the first steps of the first two systems find
    # room beside at most one other stream
    assert min(n[:2]) >= 1 + 5 and min(n[2:]) >= 5 + 5
    assert kernels_of_last_step(cglib, systems[:1]) == [2]
