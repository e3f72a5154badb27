"""Particles concentrated in small parts of the box (isolated haloes, coincident particles): the key sort's
long runs of equal upper bits and the tree's wide levels far below the mean spacing. Keys and
permutation equal numpy's stable sort, the tree the oracle's; and neither phase takes many times as long
as for a uniform box of the same size (device times from the simulation's phase events; the bounds
lie between what the phases take when these inputs use the whole chip, 2 times the uniform box's, and when they
fall to a few SMs, 8 to 90 times)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def with_runs(n, lengths, width, seed=1):
    """n particles in random order: for each length as many particles in one cube of that width, the rest uniform."""
    rng = np.random.default_rng(seed)
    x = rng.uniform(0, 1, (n, 3))
    at = 0
    for k, length in enumerate(lengths):
        cell = (rng.permutation(2048)[:3] + 0.5) / 2048  # the middle of a level-11 cube
        x[at:at + length] = cell + width * rng.uniform(-0.5, 0.5, (length, 3))
        at += length
    assert at <= n
    return x[rng.permutation(n)].astype(np.float32)


EDGES = [255, 256, 257, 511, 513, 2047, 2049, 4095, 4096, 4097, 6144, 6145, 12289]


@pytest.mark.parametrize("n", [sum(EDGES), 65536, 65537, 100003])
@pytest.mark.parametrize("width", [0.0, 1e-6, 2e-4])
def test_runs_of_every_kind_are_sorted(cpm, n, width):
    """Run lengths on both sides of those at which the method changes, below and above 65,536 keys."""
    keys, perm = cpm.octant_keys(with_runs(n, EDGES, width), 1.0)
    assert np.array_equal(perm, np.argsort(keys, kind="stable").astype(np.uint32))


@pytest.mark.parametrize("n,lengths", [(30000, [29999]), (300000, [300000]), (500000, [1000] * 400),
                                       (500000, [5000] * 99), (700001, [4097, 600000, 4096])])
def test_most_particles_in_long_runs(cpm, n, lengths):
    for width in (0.0, 1e-4):
        keys, perm = cpm.octant_keys(with_runs(n, lengths, width), 1.0)
        assert np.array_equal(perm, np.argsort(keys, kind="stable").astype(np.uint32))


def phases(cpm, x, split):
    """Mean device ms per step of each phase over four steps of a resting box."""
    nat = cpm._native
    sim = cpm.Simulation(cpm.Cosmology(0.0, 0.3, 0.7, 70.0), 1.0, 32, x, np.zeros_like(x), 0.5, split,
                         flags=nat.SIM_TIMING | nat.SIM_NO_AUTOTUNE)
    ms, steps, a = np.zeros(8), C.c_uint64(), 0.5
    for k in range(6):
        a *= 1.0000001
        sim.step_to(a)
        if k == 1:
            nat.lib().cpm_sim_phase_times(sim.h, C.c_void_p(ms.ctypes.data), C.byref(steps), 1)
    nat.lib().cpm_sim_phase_times(sim.h, C.c_void_p(ms.ctypes.data), C.byref(steps), 1)
    assert steps.value == 4
    sim.close()
    return dict(sort=ms[1], build=ms[5])


@pytest.mark.parametrize("n", [65536, 1000000])
def test_sort_time_of_a_concentrated_box(cpm, n):
    rng = np.random.default_rng(3)
    uniform = phases(cpm, rng.uniform(0, 1, (n, 3)).astype(np.float32), None)["sort"]
    for x in (0.3 + 1e-4 * rng.standard_normal((n, 3)), np.full((n, 3), 0.25)):
        assert phases(cpm, x.astype(np.float32), None)["sort"] < 6.0 * uniform


def haloes(n, members, sigma, seed=5):
    rng = np.random.default_rng(seed)
    centres = rng.uniform(0.1, 0.9, (max(1, n // members), 3))
    return (centres[rng.integers(0, len(centres), n)] + sigma * rng.standard_normal((n, 3))).astype(np.float32)


def test_tree_of_wide_deep_levels_is_the_oracles(cpm, orc):
    """400,000 particles in haloes of 10,000, each smaller than a level-12 cube: levels of tens of thousands of
    nodes from there on, after narrow ones."""
    x = haloes(400000, 10000, 2e-5)
    stats = {}
    got = cpm.tree_accelerations(x, 1.0, cpm.ForceSplit(5e-7, 2e-6, 1e-7, 0.5), 1.0, stats=stats).astype(np.float64)
    tree = orc.tree_build(x, 1.0)
    assert stats["nodes"] == len(tree["count"])
    ref = orc.tree_accelerations_com64(x, 1.0, orc.Split(5e-7, 2e-6, 1e-7, 0.5), 1.0).astype(np.float64)
    assert np.sqrt(((got - ref) ** 2).sum()) <= 1e-5 * np.sqrt((ref ** 2).sum())


def test_build_time_of_a_concentrated_box(cpm):
    n = 4000000
    split = cpm.ForceSplit(1e-6, 4e-6, 1e-7, 0.5)
    uniform = phases(cpm, np.random.default_rng(4).uniform(0, 1, (n, 3)).astype(np.float32), split)["build"]
    assert phases(cpm, haloes(n, 1500, 5e-5), split)["build"] < 4.0 * uniform
