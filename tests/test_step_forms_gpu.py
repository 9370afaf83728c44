"""The forms of an SPP step against one another at the sizes where the choice changes: runs (one launch with
the 8-lane or the thread-per-cell force pass, two launches, two launches and an integrator of its own)
and single steps from host buffers (the same forms and the step graph), each against plain kernels
(CG_GRAPH_UNROLLED=1) from the same state with the same normals, drawn or supplied.

With fixed-point sums the bits are equal. With floating-point sums positions agree to 1e-10 after six
steps of dt 0.01 of a well-conditioned tissue: forces of order 1 differ by some 1e-14 in the order of
their sums, times mu dt per step and a growth of less than 10 per step; directors do not depend on the
forces and are equal. In mixed precision positions that differ in their last bits move FP32 roundings
(6e-8 of terms up to 10): 1e-6."""
import ctypes as C

import numpy as np
import pytest

from helpers import jittered_lattice

pytestmark = pytest.mark.gpu
STEPS = 6


def make(sizes, opts):
    import cellgpu_b200 as cg

    pts, boxes = zip(*[jittered_lattice(nx, ny, 0.25, 3 + i) for i, (nx, ny) in enumerate(sizes)])
    n = sum(len(p) for p in pts)
    rng = np.random.default_rng(n)
    b = cg.VoronoiBatch([len(p) for p in pts], boxes, precision=cg.CG_MIXED if "mixed" in opts else cg.CG_FP64)
    b.set_positions(np.concatenate(pts))
    b.set_directors(rng.uniform(0, 2 * np.pi, n))
    pref = np.stack([np.ones(n), rng.uniform(3.6, 4.0, n)], 1)
    b.set_preferences(pref)
    b.set_motility(np.tile([0.3, 1.0], (n, 1)))
    b.set_seed(99)
    b.set_deterministic("deterministic" in opts)
    b.triangulate()
    return b, n, rng, pref


def same(b, ref, boxes, opts):
    assert np.array_equal(b.directors(), ref.directors())
    if "deterministic" in opts:
        assert np.array_equal(b.positions(), ref.positions())
        return
    L = np.repeat(np.asarray(boxes), ref.N, axis=0)
    d = b.positions() - ref.positions()
    d -= np.round(d / L) * L
    assert np.abs(d).max() < (1e-6 if "mixed" in opts else 1e-10)


# 28392 and 28500 cells: the last of the 8-lane pass and the first of the thread-per-cell pass in one launch;
# 81920 / 82000: one launch and two; 299000 / 301000: integration in the tail and after it; two uneven
# instances above that; other modes on both sides of 30000
@pytest.mark.parametrize("sizes,opts", [([(182, 156)], ""), ([(190, 150)], ""), ([(320, 256)], ""), ([(328, 250)], ""),
                                        ([(598, 500)], ""), ([(602, 500)], ""), ([(602, 500), (21, 20)], ""),
                                        ([(200, 150)], "mixed"), ([(201, 150)], "mixed"),
                                        ([(200, 150)], "deterministic"), ([(201, 150)], "deterministic"),
                                        ([(640, 480)], "deterministic")])
@pytest.mark.parametrize("drawn", [True, False])
def test_runs(cglib, torch, monkeypatch, sizes, opts, drawn):
    b, n, rng, pref = make(sizes, opts)
    ref = make(sizes, opts)[0]
    noise = None if drawn else torch.tensor(rng.standard_normal((STEPS, n)), device="cuda:0")
    b.spp_run(STEPS, dt=0.01, noise=noise)
    monkeypatch.setenv("CG_GRAPH_UNROLLED", "1")
    ref.spp_run(STEPS, dt=0.01, noise=noise)
    same(b, ref, b.boxes, opts)
    assert b.counters()["rows_changed"] == ref.counters()["rows_changed"] > 0


# one launch, two launches, the step graph, two launches and an integrator of its own
@pytest.mark.parametrize("sizes,opts", [([(256, 256)], ""), ([(260, 256)], ""), ([(450, 440)], ""), ([(460, 440)], ""),
                                        ([(300, 298)], "mixed"), ([(310, 298)], "mixed"),
                                        ([(300, 298)], "deterministic"), ([(310, 298)], "deterministic"),
                                        ([(128, 128)], "mixed"), ([(129, 128)], "mixed"),
                                        ([(362, 362)], "deterministic"), ([(363, 362)], "deterministic")])
@pytest.mark.parametrize("drawn", [True, False])
def test_single_steps(cglib, oracle, torch, monkeypatch, sizes, opts, drawn):
    b, n, rng, pref = make(sizes, opts)
    ref = make(sizes, opts)[0]
    noise = rng.standard_normal((STEPS, n))
    host, energy = torch.from_numpy(noise).pin_memory(), torch.zeros(STEPS, 1, dtype=torch.float64).pin_memory()
    AP = oracle.voronoi_geometry(b.positions(), b.boxes[0], *oracle.periodic_delaunay(b.positions(), b.boxes[0], 16))
    first = oracle.voronoi_energy(AP, pref)
    for t in range(STEPS):
        if drawn:
            assert cglib.cg_spp_enqueue(b.handle, 1, 0.01, 1.0) == 0
        else:
            assert cglib.cg_spp_enqueue_host(b.handle, host[t].data_ptr(), 0.01, 1.0, energy[t].data_ptr()) == 0
    done, halted = C.c_int(0), C.c_int(0)
    assert cglib.cg_poll(b.handle, C.byref(done), C.byref(halted), 0) == 0
    assert (done.value, halted.value) == (STEPS, 0)
    monkeypatch.setenv("CG_GRAPH_UNROLLED", "1")
    ref.spp_run(STEPS - 1, dt=0.01, noise=None if drawn else torch.tensor(noise[:-1], device="cuda:0"))
    ref.enforce_topology()
    ref.compute_forces()
    last = ref.energies()[0]  # of the configuration that the last step starts from
    ref.spp_run(1, dt=0.01, noise=None if drawn else torch.tensor(noise[-1:], device="cuda:0"))
    same(b, ref, b.boxes, opts)
    if not drawn:
        rtol = 1e-5 if opts == "mixed" else 1e-11
        assert abs(energy[0, 0].item() - first) < rtol * first
        assert abs(energy[-1, 0].item() - last) < rtol * last


# FIRE in cooperative launches with the 8-lane and the thread-per-cell pass, against plain kernels
@pytest.mark.parametrize("nx,ny", [(182, 156), (190, 150), (446, 440)])
def test_fire(cglib, monkeypatch, nx, ny):
    import cellgpu_b200 as cg

    prm = cg.FireParams.defaults(force_cutoff=1e-12, max_iterations=20)
    b = make([(nx, ny)], "")[0]
    ref = make([(nx, ny)], "")[0]
    b.fire_minimize(prm)
    monkeypatch.setenv("CG_GRAPH_UNROLLED", "1")
    ref.fire_minimize(prm)
    assert b.fire_state()[0][0] == ref.fire_state()[0][0] == 20
    d = b.positions() - ref.positions()
    d -= np.round(d / b.boxes[0]) * b.boxes[0]
    assert np.abs(d).max() < 1e-10


@pytest.fixture(scope="module")
def torch():
    import torch
    return torch
