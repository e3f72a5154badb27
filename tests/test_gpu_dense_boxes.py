"""Which walk serves which box: a simulation's dense boxes take the ordered walk, with and without a list of
walked particles, and every other box and call the group walk. The two add a particle's terms in different orders,
so their sums agree to rounding and differ in some last bit: bit equality tells which one ran."""
import numpy as np
import pytest

import net_oracle as no
from test_gpu_walk import BOX, dense

pytestmark = pytest.mark.gpu

SPLIT = (0.35, 1.5, 0.02, 0.5)


def rel_rms(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return float(np.sqrt(((a - b) ** 2).sum() / (b ** 2).sum()))


def simulation(cpm, x, mesh=64):
    return cpm.Simulation(cpm.Cosmology(0.0, 0.3, 0.7, 70.0), BOX, mesh, x, np.zeros_like(x), 0.5,
                          cpm.ForceSplit(*SPLIT), flags=cpm._native.SIM_NO_AUTOTUNE)


def is_dense(sim):
    spread = 0
    while sim.n >> (3 * spread) > 1:
        spread += 1
    return sim.tree_depth()["max_depth"] > spread + 4


def test_dense_boxes_and_only_they_take_the_ordered_walk(cpm):
    for x, want in ((dense(20000), True), (np.random.default_rng(2).uniform(0, BOX, (20000, 3)).astype(np.float32) % np.float32(BOX), False)):
        sim = simulation(cpm, x)
        assert is_dense(sim) == want
        k = 1.5 * 0.3 * BOX ** 3 / (4.0 * np.pi * 0.5 * len(x))
        sr, call = sim.short_range(), cpm.tree_accelerations(x, BOX, cpm.ForceSplit(*SPLIT), k)
        assert rel_rms(sr, call) < 1e-5
        ratio = sr.astype(np.float64) / np.where(call == 0, 1, call)  # the coupling's rounding is common to all
        common = np.median(ratio)
        same = np.mean(np.abs(ratio / common - 1.0) < 1.0e-7)
        assert (same < 0.9) if want else (same == 1.0)
        sim.close()


def test_learned_step_with_every_particle_dense_equals_plain_step_in_a_dense_box(cpm):
    """The list of all particles in the sorted order: the walk over it is the plain walk, bit for bit."""
    x = dense(20000)
    net = cpm.ShortRangeNet(64, no.random_weights(3))
    plain, learned = simulation(cpm, x), simulation(cpm, x)
    learned.set_learned(net, -1e30)
    a = 0.5
    for _ in range(6):
        a = float(np.float32(a * 1.001))
        plain.step_to(a)
        learned.step_to(a)
    assert is_dense(plain) and learned.walked() == len(x)
    p, q = plain.state(), learned.state()
    for key in ("x", "p", "acc"):
        assert np.array_equal(p[key], q[key]), key
    for s in (plain, learned):
        s.close()
    net.close()


def test_list_walks_of_dense_boxes(cpm, orc):
    """A list that leaves most particles out: the walked ones get the force of the plain step's walk."""
    x = dense(33333)
    net = cpm.ShortRangeNet(64, no.random_weights(3, scale=0.0))  # serves a zero field
    sim = simulation(cpm, x)
    assert is_dense(sim)
    pm = sim.state()["acc"].astype(np.float64) - sim.short_range()
    sim.set_learned(net, 30.0)
    sim.set_state(x, np.zeros_like(x))
    assert 0 < sim.walked() < len(x) // 2
    sr = sim.state()["acc"].astype(np.float64) - pm
    walked = np.abs(sr).max(axis=1) > 1e-6 * np.abs(sr).max()
    k = 1.5 * 0.3 * BOX ** 3 / (4.0 * np.pi * 0.5 * len(x))
    ref = orc.tree_accelerations_com64(x, BOX, orc.Split(*SPLIT), k).astype(np.float64)
    assert rel_rms(sr[walked], ref[walked]) < 1e-5
    sim.close()
    net.close()


def test_boxes_of_a_batch_take_their_own_walk(cpm):
    """Dense and other boxes side by side in one batch (run well past z = 0): each box's force is that of a
    simulation of its own in the same state."""
    cc, box, n_side, mesh, boxes = cpm.Cosmology(0.0, 0.3, 0.7, 70.0), 16.0, 32, 64, 6
    split = cpm.ForceSplit.with_(box, mesh, n_side, 1.0 / 30.0, 0.5)
    fixed = cpm._native.SIM_NO_AUTOTUNE
    ens = cpm.Ensemble(cc, box, 0.96, 0.8, 0.02, [(n_side, mesh, boxes, 40, split)], flags=fixed)
    mixed = 0
    for k, a in enumerate(cpm.ln_a_schedule(0.02, 3.0, 128)[:115]):
        ens.step_to(a)
        if k < 106 or k % 2:
            continue
        marks = []
        for b in range(boxes):
            e = ens.state(0, b)
            single = cpm.Simulation(cc, box, mesh, e["x"], e["p"], a, split, flags=fixed)
            assert rel_rms(e["acc"], single.state()["acc"]) < 1e-5, (a, b)
            marks.append(is_dense(single))
            single.close()
        mixed += any(marks) and not all(marks)
    assert mixed
    ens.close()
