"""T1 sweeps that stop at a full cell row in batches of more instances than the GPU runs at once: the
other instances, those whose blocks start afterwards among them, finish their sweep in the same launch;
the rows grow, the stopped sweeps resume, and every instance ends as the reference's sequential sweep."""
import numpy as np
import pytest

from helpers import jittered_lattice

pytestmark = pytest.mark.gpu

THRESHOLD = 0.45


def batch(oracle, sizes):
    import cellgpu_b200 as cg

    st = []
    for i, (nx, ny) in enumerate(sizes):
        pos, box = jittered_lattice(nx, ny, 0.3, 40 + i)
        st.append((pos, box, oracle.vertex_from_delaunay(pos, box, *oracle.periodic_delaunay(pos, box, 16), vmax=30)))
    vmax = max(int(w[3].max()) for _, _, w in st)  # no room for another vertex in the widest rows
    b = cg.VertexBatch([len(p) for p, _, _ in st], [box for _, box, _ in st], vmax=vmax)
    cat = lambda k, per: np.concatenate([w[k] + per * int(o) for (_, _, w), o in zip(st, b.offsets)])
    b.set_positions(np.concatenate([w[0] for _, _, w in st]))
    b.set_vertex_topology(cat(1, 2), cat(2, 1), cat(3, 0), np.concatenate(
        [np.where(w[4] >= 0, w[4] + 2 * int(o), -1)[:, :vmax] for (_, _, w), o in zip(st, b.offsets)]))
    b.set_preferences(np.tile([1.0, 3.85], (b.Ntot, 1)))
    b.set_t1_threshold(THRESHOLD)
    return b, st, vmax


def same_wiring(b, st):
    gvn, gvcn, gcvn, gcv = b.vertex_topology()
    for i, (_, _, (_, vn, vcn, cvn, cv)) in enumerate(st):
        c0, c1 = int(b.offsets[i]), int(b.offsets[i + 1])
        assert np.array_equal(gvn[6 * c0:6 * c1] - 2 * c0, vn)
        assert np.array_equal(gvcn[6 * c0:6 * c1] - c0, vcn)
        assert np.array_equal(gcvn[c0:c1], cvn)
        for c in range(c1 - c0):
            assert np.array_equal(gcv[c0 + c, :cvn[c]] - 2 * c0, cv[c, :cvn[c]])


# a large instance first (its sweep outlasts many others) and last
@pytest.mark.parametrize("sizes", [[(25, 20)] + [(6, 6)] * 300, [(8, 6)] * 200 + [(30, 30)]])
def test_every_instance_finishes_its_sweep(oracle, sizes):
    b, st, vmax = batch(oracle, sizes)
    b.enforce_topology()
    assert b.row_capacity() > vmax
    flips = sum(len(oracle.vertex_t1(w[0], box, THRESHOLD, *w[1:], max_events=100000)) for _, box, w in st)
    same_wiring(b, st)
    assert b.counters()["t1_flips"] == flips
    assert np.array_equal(b.positions(), np.concatenate([w[0] for _, _, w in st]))


def test_steps_of_a_batch(oracle):
    import torch

    b, st, vmax = batch(oracle, [(25, 20)] + [(6, 6)] * 180)
    steps = 4
    noise = np.random.default_rng(3).normal(size=(steps, b.Nv, 2))
    b.brownian_run(steps, dt=0.01, mu=1.0, T=0.02, noise=torch.tensor(noise.reshape(steps, -1), device="cuda:0"))
    assert b.row_capacity() > vmax
    flips = 0
    for i, (_, box, (vpos, vn, vcn, cvn, cv)) in enumerate(st):
        v0 = 2 * int(b.offsets[i])
        pref = np.tile([1.0, 3.85], (len(cvn), 1))
        _, _, k = oracle.vertex_brownian_run(vpos, box, vn, vcn, cvn, cv, pref, noise[:, v0:v0 + len(vpos)], dt=0.01,
                                             T=0.02, t1_threshold=THRESHOLD)
        flips += k
        assert np.abs(b.positions()[v0:v0 + len(vpos)] - vpos).max() < 1e-9
    same_wiring(b, st)
    assert b.counters()["t1_flips"] == flips
