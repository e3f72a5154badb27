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
