"""Systems whose cooperative launches the driver refuses (more blocks than the GPU holds; nothing of such a
launch runs) step and minimise by graphs: the bits of an ordinary run with fixed-point sums, 1e-10 after
a few iterations of FIRE and vertex steps with floating-point ones."""
import numpy as np
import pytest

from helpers import jittered_lattice

pytestmark = pytest.mark.gpu


def voronoi(nx, ny, det=True):
    import cellgpu_b200 as cg

    pos, box = jittered_lattice(nx, ny, 0.3, 4)
    n = len(pos)
    b = cg.VoronoiBatch([n], [box])
    b.set_positions(pos)
    b.set_directors(np.linspace(0, 6, n))
    b.set_motility(np.tile([0.2, 1.0], (n, 1)))
    b.set_preferences(np.tile([1.0, 3.8], (n, 1)))
    b.set_seed(5)
    b.set_deterministic(det)
    b.triangulate()
    return b


def vertex():
    import cellgpu_b200 as cg

    pos, box = jittered_lattice(20, 15, 0.3, 4)
    b = cg.VertexBatch([len(pos)], [box])
    b.from_cells(pos)
    b.set_preferences(np.tile([1.0, 3.8], (len(pos), 1)))
    b.set_t1_threshold(0.04)
    b.set_seed(5)
    return b


def enqueue(b):
    for n in (1, 7):
        assert b._lib.cg_spp_enqueue(b.handle, n, 0.01, 1.0) == 0
    assert b._lib.cg_synchronize(b.handle) == 0


def host(b):
    import torch

    noise = torch.from_numpy(np.random.default_rng(1).standard_normal((4, b.Ntot))).pin_memory()
    energy = torch.zeros(4, 1, dtype=torch.float64).pin_memory()
    for t in range(4):
        assert b._lib.cg_spp_enqueue_host(b.handle, noise[t].data_ptr(), 0.01, 1.0, energy[t].data_ptr()) == 0
    assert b._lib.cg_synchronize(b.handle) == 0
    b.energy_log = energy.numpy().copy()


def fire(b):
    import cellgpu_b200 as cg

    b.fire_minimize(cg.FireParams.defaults(force_cutoff=1e-12, max_iterations=24))


@pytest.mark.parametrize("make,run,exact", [(lambda: voronoi(20, 15), lambda b: b.spp_run(40), True),
                                            (lambda: voronoi(96, 100), lambda b: b.spp_run(40), True),
                                            (lambda: voronoi(182, 182), lambda b: b.spp_run(10), True),
                                            (lambda: voronoi(182, 182), enqueue, True),
                                            (lambda: voronoi(33, 32), host, True),
                                            (lambda: voronoi(33, 32, False), host, False),
                                            (lambda: voronoi(260, 256, False), host, False),
                                            (lambda: voronoi(20, 15, False), fire, False),
                                            (vertex, lambda b: b.brownian_run(10), False), (vertex, fire, False)])
def test_steps_run_by_graphs(cglib, make, run, exact):
    a, b = make(), make()
    assert cglib.cg_inject_refusal(b.handle, 1) == 0
    for _ in range(2):  # the second call finds the system refused
        run(a)
        run(b)
    if exact:
        assert np.array_equal(a.positions(), b.positions())
    else:
        d = a.positions() - b.positions()
        d -= np.round(d / a.boxes[0]) * a.boxes[0]
        assert np.abs(d).max() < 1e-10
    if run is host:
        np.testing.assert_allclose(b.energy_log, a.energy_log, rtol=1e-11)
    # a later refusal-free launch is not tried again, and the context is as before
    assert cglib.cg_inject_refusal(b.handle, 0) == 0
    run(b)
