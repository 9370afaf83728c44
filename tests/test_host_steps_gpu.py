"""Host-driven steps overlap their copies: the noise of the next step is copied in beside the step that runs,
so a host step takes no longer than one whose normals are drawn (0.97 of it, reading them being cheaper;
1.11 where the clearing of the force sums waits behind the copy). The bound is halfway."""
import ctypes as C
import time

import numpy as np
import pytest

from helpers import jittered_lattice

pytestmark = pytest.mark.gpu


def test_copies_overlap_steps(cglib):
    import torch
    import cellgpu_b200 as cg

    pos, box = jittered_lattice(300, 300, 0.3, 2)
    n, steps = len(pos), 40
    pos = pos[np.random.default_rng(1).permutation(n)]
    b = cg.VoronoiBatch([n], [box])
    b.set_positions(pos)
    b.set_directors(np.zeros(n))
    b.set_motility(np.tile([0.05, 1.0], (n, 1)))
    b.set_preferences(np.tile([1.0, 3.8], (n, 1)))
    b.triangulate()
    noise = torch.from_numpy(np.random.default_rng(0).standard_normal((steps, n))).pin_memory()
    done, halted = C.c_int(0), C.c_int(0)

    def timed(step):
        t0 = time.perf_counter()
        for t in range(steps):
            assert step(t) == 0
        assert cglib.cg_poll(b.handle, C.byref(done), C.byref(halted), 1) == 0
        return time.perf_counter() - t0

    host = lambda t: cglib.cg_spp_enqueue_host(b.handle, noise[t].data_ptr(), 0.01, 1.0, None)
    drawn = lambda t: cglib.cg_spp_enqueue(b.handle, 1, 0.01, 1.0)
    timed(host), timed(drawn)
    assert min(timed(host) for _ in range(8)) < 1.04 * min(timed(drawn) for _ in range(8))
