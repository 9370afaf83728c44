"""Host steps whose energies go to page-locked memory, across a halt: the step before it, the step that
halts and the steps enqueued after it all store the energies of the areas and perimeters that the system
holds, whatever form runs them, and after the recovery the steps go on."""
import ctypes as C

import numpy as np
import pytest

from helpers import jittered_lattice

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,opts", [([(20, 15)], ""), ([(33, 32)], ""), ([(20, 15), (40, 41), (25, 24)], ""),
                                        ([(96, 100)], "mixed"), ([(260, 256)], ""), ([(260, 256)], "mixed"),
                                        ([(33, 33)], "deterministic"), ([(260, 256)], "deterministic")])
def test_energies_across_a_halt(cglib, oracle, sizes, opts):
    import torch
    import cellgpu_b200 as cg

    pts, boxes = zip(*[jittered_lattice(nx, ny, 0.3, 5 + i) for i, (nx, ny) in enumerate(sizes)])
    n = sum(len(p) for p in pts)
    rng = np.random.default_rng(n)
    b = cg.VoronoiBatch([len(p) for p in pts], boxes, precision=cg.CG_MIXED if opts == "mixed" else cg.CG_FP64)
    b.set_positions(np.concatenate(pts))
    b.set_directors(rng.uniform(0, 2 * np.pi, n))
    b.set_preferences(np.tile([1.0, 3.8], (n, 1)))
    b.set_motility(np.tile([1.5, 1.0], (n, 1)))  # with dt = 1 every cell leaves its neighbours
    b.set_deterministic(opts == "deterministic")
    b.triangulate()
    noise = torch.from_numpy(rng.standard_normal((4, n))).pin_memory()
    energy = torch.full((4, len(pts)), -1.0, dtype=torch.float64).pin_memory()
    step = lambda t: cglib.cg_spp_enqueue_host(b.handle, noise[t].data_ptr(), 1.0, 0.0, energy[t].data_ptr())
    for t in range(3):
        assert step(t) == 0
    done, halted = C.c_int(0), C.c_int(0)
    assert cglib.cg_poll(b.handle, C.byref(done), C.byref(halted), 0) == 0
    assert (done.value, halted.value) == (1, 1)
    first = []
    for p, box in zip(pts, boxes):
        AP = oracle.voronoi_geometry(p, box, *oracle.periodic_delaunay(p, box, 16))
        first.append(oracle.voronoi_energy(AP, np.tile([1.0, 3.8], (len(p), 1))))
    np.testing.assert_allclose(energy[0].numpy(), first, rtol=1e-5 if opts == "mixed" else 1e-11)
    held = b.energies()  # sums of the same terms in another order
    for t in (1, 2):
        np.testing.assert_allclose(energy[t].numpy(), held, rtol=1e-9)
    assert cglib.cg_poll(b.handle, C.byref(done), C.byref(halted), 1) == 0
    assert step(3) == 0
    assert cglib.cg_poll(b.handle, C.byref(done), C.byref(halted), 0) == 0
    assert (done.value, halted.value) == (2, 0)
    assert np.isfinite(energy[3].numpy()).all()
