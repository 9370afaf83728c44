"""Host-driven steps of large systems clear their force sums in a kernel of their own (a memset would wait for
the copy of the next step's noise that runs beside the step), small ones, one cluster, by a memset."""
import ctypes as C

import numpy as np
import pytest

from helpers import jittered_lattice

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,kernels", [(20, 15, 1), (33, 32, 2), (300, 300, 3)])  # one cluster, one launch, two launches
def test_kernels_of_a_host_step(cglib, nx, ny, kernels):
    import torch
    import cellgpu_b200 as cg

    pos, box = jittered_lattice(nx, ny, 0.2, 2)
    n, steps = len(pos), 5
    b = cg.VoronoiBatch([n], [box])
    b.set_positions(pos)
    b.set_directors(np.zeros(n))
    b.set_motility(np.tile([0.05, 1.0], (n, 1)))
    b.set_preferences(np.tile([1.0, 3.8], (n, 1)))
    b.triangulate()
    noise = torch.from_numpy(np.random.default_rng(0).standard_normal((steps, n))).pin_memory()
    before = cglib.cg_kernels_launched(b.handle)
    for t in range(steps):
        assert cglib.cg_spp_enqueue_host(b.handle, noise[t].data_ptr(), 0.01, 1.0, None) == 0
    done, halted = C.c_int(0), C.c_int(0)
    assert cglib.cg_poll(b.handle, C.byref(done), C.byref(halted), 0) == 0
    assert (done.value, halted.value) == (steps, 0)
    assert cglib.cg_kernels_launched(b.handle) - before == kernels * steps
