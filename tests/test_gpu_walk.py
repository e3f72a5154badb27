"""The tree walk where its group-level decisions can go wrong, against the oracle's walk with FP64
centres of mass (the GPU's): periodic images of every kind (cutoffs up to and beyond half the box,
positions outside it), degenerate cutoffs, and group counts on both sides of the team sizes. Pair and
accept counts are those of the oracle; accelerations lie within the tree's 1e-5 relative RMS."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOX = 10.0


def clumped(n, seed):
    """Half uniform, half in clumps of width 0.1 that lie anywhere, box faces and corners included."""
    rng = np.random.default_rng(seed)
    x = rng.uniform(0, BOX, (n, 3))
    centres = np.concatenate([rng.uniform(0, BOX, (40, 3)), [[0.0, 0.0, 0.0], [0.0, 5.0, 9.99]]])
    m = n // 2
    x[:m] = centres[rng.integers(0, len(centres), m)] + 0.1 * rng.standard_normal((m, 3))
    return np.float32(np.mod(x, BOX)) % np.float32(BOX)


def check(cpm, orc, x, split):
    stats = {}
    got = cpm.tree_accelerations(x, BOX, cpm.ForceSplit(*split), 1.0, stats=stats).astype(np.float64)
    ref = orc.tree_accelerations_com64(x, BOX, orc.Split(*split), 1.0).astype(np.float64)
    assert np.all(np.isfinite(got))
    assert np.sqrt(((got - ref) ** 2).sum()) <= 1e-5 * np.sqrt((ref ** 2).sum())
    if split[3] == 0.0:  # no node is accepted: the counts hang on exact tests only
        pairs, accepts, _ = orc.tree_walk_stats(x, BOX, orc.Split(*split))
        assert stats["leaf_pairs"] == pairs and stats["node_accepts"] == accepts == 0


@pytest.mark.parametrize("theta", [0.0, 0.5])
@pytest.mark.parametrize("r_cut", [0.0, 0.3, 2.5, 4.9, 5.0, 8.0])
def test_cutoffs_against_the_box(cpm, orc, r_cut, theta):
    check(cpm, orc, clumped(4000, 3), (0.5, r_cut, 0.05, theta))


@pytest.mark.parametrize("theta", [0.0, 0.5])
def test_positions_outside_the_box(cpm, orc, theta):
    """The octant descent takes any finite position; its cube then does not hold the particle."""
    x = clumped(5000, 5)
    x[::7] += np.float32(BOX) * np.float32([1.0, 0.0, -1.0])
    x[::11, 1] -= np.float32(3.0 * BOX)
    check(cpm, orc, x, (0.4, 1.5, 0.05, theta))


def test_edges_of_the_box(cpm, orc):
    """Coordinates exactly 0, L and L/2: cube faces and corners."""
    g = np.float32([0.0, 2.5, 5.0, 7.5, BOX])
    x = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    check(cpm, orc, np.concatenate([x, clumped(500, 6)]), (0.6, 2.6, 0.05, 0.5))


# One warp per group, teams of 2 and teams of 4 (the group counts 7104 and 3552 are the last of each),
# full and ragged groups, trees that are one leaf.
@pytest.mark.parametrize("n", [1, 8, 9, 33, 3552 * 32, 3552 * 32 + 1, 7104 * 32, 7104 * 32 + 33])
def test_group_counts(cpm, orc, n):
    check(cpm, orc, clumped(n, 7), (0.12, 0.4, 0.01, 0.5))


def dense(n):
    """clumped() with a core at a corner of the box and one inside it."""
    x = clumped(n, 9)
    rng, m = np.random.default_rng(10), n // 5
    x[:m] = np.mod(0.005 * rng.standard_normal((m, 3)) + np.array([[0.0], [7.3]])[np.arange(m) % 2], BOX)
    return x % np.float32(BOX)


def dense_simulation(cpm, x, split, flags):
    cc = cpm.Cosmology(0.0, 0.3, 0.7, 70.0)
    sim = cpm.Simulation(cc, BOX, 32, x, np.zeros_like(x), 0.5, cpm.ForceSplit(*split), flags=flags)
    depth, spread = sim.tree_depth()["max_depth"], 0
    while len(x) >> (3 * spread) > 1:
        spread += 1
    assert depth >= spread + 4
    return sim


@pytest.mark.parametrize("n,r_cut", [(500, 1.5), (4000, 4.0), (4000, 8.0), (33333, 0.7)])
def test_dense_simulations_walk_in_order(cpm, orc, n, r_cut):
    """A simulation whose tree is deep takes the ordered walk, the function call does not: both are the
    oracle's force, of the same pairs and accepts."""
    x, split = dense(n), (0.35, r_cut, 0.02, 0.5)
    sim = dense_simulation(cpm, x, split, 0)
    k = 1.5 * 0.3 * BOX ** 3 / (4.0 * np.pi * 0.5 * n)
    sr = sim.short_range().astype(np.float64)
    ref = orc.tree_accelerations_com64(x, BOX, orc.Split(*split), k).astype(np.float64)
    assert np.sqrt(((sr - ref) ** 2).sum()) <= 1e-5 * np.sqrt((ref ** 2).sum())
    stats = {}
    cpm.tree_accelerations(x, BOX, cpm.ForceSplit(*split), k, stats=stats)
    counters = sim.counters()
    assert (counters["leaf_pairs"], counters["node_accepts"]) == (stats["leaf_pairs"], stats["node_accepts"])
    sim.close()


def test_dense_simulations_with_quadrupoles(cpm, orc):
    """Quadrupole terms in the ordered walk: none where no node is accepted (theta = 0), and at theta 0.5
    a smaller error against the sum over all pairs than without them."""
    x, nat = dense(4000), cpm._native
    exact = orc.tree_accelerations_com64(x, BOX, orc.Split(0.35, 1.5, 0.02, 0.0),
                                         1.5 * 0.3 * BOX ** 3 / (4.0 * np.pi * 0.5 * len(x))).astype(np.float64)
    sr = {}
    for theta in (0.0, 0.5):
        for flags in (0, nat.SIM_QUADRUPOLE):
            sim = dense_simulation(cpm, x, (0.35, 1.5, 0.02, theta), flags)
            sr[theta, flags] = sim.short_range().astype(np.float64)
            sim.close()
    assert np.array_equal(sr[0.0, 0], sr[0.0, nat.SIM_QUADRUPOLE])
    err = [np.sqrt(((sr[0.5, f] - exact) ** 2).sum()) for f in (0, nat.SIM_QUADRUPOLE)]
    assert err[1] < err[0]
