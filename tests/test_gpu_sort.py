"""The key sort and the tree build on both sides of every size at which they change method (one
cluster, a launch per pass or level, the scan of the tile counts) and over every kind of run that
shares the sorted upper bits: keys and permutation against numpy's stable sort, the tree against the
oracle's. Whole numbers: equality."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def positions(n, kind, seed=1):
    rng = np.random.default_rng(seed)
    x = rng.uniform(0, 1, (n, 3))
    if kind == "clump":  # long runs of equal upper bits: distinct keys, equal keys, a few and thousands
        m = n // 4
        x[:m] = 0.3 + 1e-5 * rng.uniform(0, 1, (m, 3))
        x[m:2 * m] = 0.7 + 1e-4 * rng.integers(0, 4, (m, 3))
        x[2 * m:2 * m + n // 8] = x[rng.integers(3 * m, n, n // 8)]
        x = x[rng.permutation(n)]
    elif kind == "same":
        x[:] = 0.25
    return x.astype(np.float32)


@pytest.mark.parametrize("kind", ["uniform", "clump", "same"])
@pytest.mark.parametrize("n", [1, 2, 33, 8192, 65535, 65536, 65537, 262144, 262145, 700001])
def test_sort_is_numpys_stable_sort(cpm, n, kind):
    keys, perm = cpm.octant_keys(positions(n, kind), 1.0)
    assert np.array_equal(perm, np.argsort(keys, kind="stable").astype(np.uint32))


@pytest.mark.parametrize("levels", [1, 3, 10, 11, 12, 21])
@pytest.mark.parametrize("n", [5000, 100001])
def test_sort_of_shorter_keys(cpm, n, levels):
    keys, perm = cpm.octant_keys(positions(n, "clump"), 1.0, levels)
    assert keys.max() < 1 << (3 * levels)
    assert np.array_equal(perm, np.argsort(keys, kind="stable").astype(np.uint32))


@pytest.mark.parametrize("n", [1, 8, 9, 65, 2048, 2049, 262144, 262145])
def test_tree_is_the_oracles(cpm, orc, n):
    x = positions(n, "uniform", 2)
    x[: n // 3] = np.float32(0.5) + np.float32(0.01) * (x[: n // 3] - np.float32(0.5))
    stats = {}
    got = cpm.tree_accelerations(x, 1.0, cpm.ForceSplit(0.02, 0.06, 0.001, 0.5), 1.0, stats=stats).astype(np.float64)
    tree = orc.tree_build(x, 1.0)
    assert stats["nodes"] == len(tree["count"])
    ref = orc.tree_accelerations_com64(x, 1.0, orc.Split(0.02, 0.06, 0.001, 0.5), 1.0).astype(np.float64)
    assert np.sqrt(((got - ref) ** 2).sum()) <= 1e-5 * np.sqrt((ref ** 2).sum())
