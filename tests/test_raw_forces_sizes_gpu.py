"""cg_voronoi_forces on both sides of the size where raw calls take the thread-per-cell pass (37888 cells):
the last call of the 8-lane pass, the first of the other one, and one with a partial last warp, against
the oracle."""
import ctypes as C

import numpy as np
import pytest

from helpers import force_error, jittered_lattice

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(219, 173), (256, 148), (227, 167)])
def test_forces_match_oracle(cglib, oracle, nx, ny):
    import torch

    pos, box = jittered_lattice(nx, ny, 0.35, nx)
    n = len(pos)
    nn, nbr = oracle.periodic_delaunay(pos, box, 16)
    pref = np.stack([np.ones(n), np.random.default_rng(ny).uniform(3.6, 4.0, n)], 1)
    AP = oracle.voronoi_geometry(pos, box, nn, nbr)
    F = oracle.voronoi_forces(pos, box, nn, nbr, AP, pref)
    dev = lambda x: torch.tensor(x, device="cuda:0")
    tpos, tnn, tnbr, tpref = dev(pos), dev(np.asarray(nn, np.int32)), dev(np.asarray(nbr, np.int32)), dev(pref)
    tAP, tF = torch.zeros_like(tpos), torch.zeros_like(tpos)
    p = lambda t: C.c_void_p(t.data_ptr())
    assert cglib.cg_voronoi_forces(p(tpos), p(tnn), p(tnbr), 16, n, box[0], box[1], p(tpref), 1.0, 1.0, p(tAP), p(tF),
                                   None) == 0
    torch.cuda.synchronize()
    assert force_error(tF.cpu().numpy(), F) < 1e-10
    np.testing.assert_allclose(tAP.cpu().numpy(), AP, rtol=1e-12)
