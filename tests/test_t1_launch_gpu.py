"""T1 detection and sweep of a single instance on both sides of the sizes where one launch becomes two (steps
above 40000 cells, sweeps alone and FIRE iterations above 8192): wiring and flips as the reference's
sequential sweep, positions bit-exact for a sweep alone and to the suite's 1e-10 after steps."""
import numpy as np
import pytest

from helpers import jittered_lattice

pytestmark = pytest.mark.gpu


def make(oracle, nx, ny):
    import cellgpu_b200 as cg

    pos, box = jittered_lattice(nx, ny, 0.3, 21)
    w = oracle.vertex_from_delaunay(pos, box, *oracle.periodic_delaunay(pos, box, 16), vmax=30)
    b = cg.VertexBatch([len(pos)], [box], vmax=30)
    b.set_positions(w[0])
    b.set_vertex_topology(*w[1:])
    b.set_preferences(np.tile([1.0, 3.85], (len(pos), 1)))
    b.set_t1_threshold(0.08)
    return b, box, w


def same_wiring(b, w):
    gvn, gvcn, gcvn, gcv = b.vertex_topology()
    assert np.array_equal(gvn, w[1]) and np.array_equal(gvcn, w[2]) and np.array_equal(gcvn, w[3])
    k = np.arange(gcv.shape[1]) < w[3][:, None]
    assert np.array_equal(np.where(k, gcv, -1), np.where(k, w[4], -1))


@pytest.mark.parametrize("nx,ny", [(128, 64), (129, 64)])
def test_sweep_alone(cglib, oracle, nx, ny):
    b, box, w = make(oracle, nx, ny)
    b.enforce_topology()
    flips = len(oracle.vertex_t1(w[0], box, 0.08, *w[1:], max_events=100000))
    assert flips > 10
    assert b.counters()["t1_flips"] == flips
    same_wiring(b, w)
    assert np.array_equal(b.positions(), w[0])


@pytest.mark.parametrize("nx,ny", [(200, 200), (201, 200)])
def test_steps(cglib, oracle, nx, ny):
    import torch

    b, box, w = make(oracle, nx, ny)
    steps = 3
    noise = np.random.default_rng(2).normal(size=(steps, b.Nv, 2))
    b.brownian_run(steps, dt=0.005, mu=1.0, T=1e-3, noise=torch.tensor(noise.reshape(steps, -1), device="cuda:0"))
    _, _, flips = oracle.vertex_brownian_run(w[0], box, *w[1:], np.tile([1.0, 3.85], (b.Ntot, 1)), noise, dt=0.005,
                                             T=1e-3, t1_threshold=0.08)
    assert flips > 10
    assert b.counters()["t1_flips"] == flips
    same_wiring(b, w)
    assert np.abs(b.positions() - w[0]).max() < 1e-10
