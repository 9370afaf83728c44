"""A barrier wait that gives up (failure injection: an arrival that nothing makes, a limit of 0.2 s) ends
the launch with CG_ERR_TIMEOUT in every cooperative form, the system is refused from then on, and other
systems go on."""
import numpy as np
import pytest

from helpers import jittered_lattice

pytestmark = pytest.mark.gpu


def voronoi(nx, ny, det):
    import cellgpu_b200 as cg

    pos, box = jittered_lattice(nx, ny, 0.3, 1)
    n = len(pos)
    b = cg.VoronoiBatch([n], [box])
    b.set_positions(pos)
    b.set_directors(np.zeros(n))
    b.set_motility(np.tile([0.05, 1.0], (n, 1)))
    b.set_preferences(np.tile([1.0, 3.8], (n, 1)))
    b.set_deterministic(det)
    b.triangulate()
    return b


def vertex():
    import cellgpu_b200 as cg

    pos, box = jittered_lattice(20, 15, 0.3, 1)
    b = cg.VertexBatch([len(pos)], [box])
    b.from_cells(pos)
    b.set_preferences(np.tile([1.0, 3.8], (len(pos), 1)))
    b.set_t1_threshold(0.04)
    return b


def fire(b):
    import cellgpu_b200 as cg

    b.fire_minimize(cg.FireParams.defaults(force_cutoff=1e-12, max_iterations=20))


# one launch (grids of a cluster's size and above), two launches per step, FIRE, and the vertex model's forms
@pytest.mark.parametrize("make,run", [(lambda: voronoi(20, 15, False), lambda b: b.spp_run(5)),
                                      (lambda: voronoi(96, 100, True), lambda b: b.spp_run(5)),
                                      (lambda: voronoi(182, 182, True), lambda b: b.spp_run(5)),
                                      (lambda: voronoi(20, 15, False), fire),
                                      (vertex, lambda b: b.brownian_run(5)),
                                      (vertex, fire)])
def test_wait_that_gives_up(cglib, make, run):
    from cellgpu_b200 import CG_ERR_TIMEOUT, CellGPUError

    b, other = make(), make()
    assert cglib.cg_inject_stall(b.handle, 0.2) == 0
    for limit in (0.2, 0.0):  # refused also once the waits would end
        assert cglib.cg_inject_stall(b.handle, limit) == 0
        for call in (run, fire, lambda x: x.compute_forces()):
            with pytest.raises(CellGPUError) as e:
                call(b)
            assert e.value.code == CG_ERR_TIMEOUT
    run(other)
    assert np.isfinite(other.positions()).all()


def test_limit_is_checked(cglib):
    b = vertex()
    for bad in (-1.0, 11.0, float("nan")):
        assert cglib.cg_inject_stall(b.handle, bad) == -2
