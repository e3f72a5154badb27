"""The walks' sets of interactions, exactly: on positions whose coordinate sums are exact in f32 in any order, so that the
centres of mass are the reference's to the last bit, both walks sum the pairs and accept the nodes that the
oracle's walk does, at opening angles where nodes are accepted."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOX, UNIT, N = 16.0, 64, 4000  # N * BOX * UNIT < 2^24


def lattice(width, seed):
    rng = np.random.default_rng(seed)
    x = rng.uniform(0, BOX, (N, 3))
    centres = np.concatenate([rng.uniform(0, BOX, (40, 3)), [[0.0, 0.0, 0.0], [0.0, 8.0, 15.9]]])
    x[:N // 2] = centres[rng.integers(0, len(centres), N // 2)] + width * rng.standard_normal((N // 2, 3))
    return (np.mod(np.round(x * UNIT), BOX * UNIT) / UNIT).astype(np.float32)


@pytest.mark.parametrize("theta", [0.3, 0.5, 0.8])
@pytest.mark.parametrize("r_cut", [0.6, 2.5, 8.5])
@pytest.mark.parametrize("width,dense", [(0.5, False), (0.04, True)])
def test_pairs_and_accepted_nodes(cpm, orc, theta, r_cut, width, dense):
    x, split = lattice(width, 11), (0.4, r_cut, 0.05, theta)
    pairs, accepts, _ = orc.tree_walk_stats(x, BOX, orc.Split(*split))
    assert pairs > 0 and (accepts > 0 or r_cut < 1.0)
    stats = {}
    cpm.tree_accelerations(x, BOX, cpm.ForceSplit(*split), 1.0, stats=stats)
    assert (stats["leaf_pairs"], stats["node_accepts"]) == (pairs, accepts)
    sim = cpm.Simulation(cpm.Cosmology(0.0, 0.3, 0.7, 70.0), BOX, 32, x, np.zeros_like(x), 0.5, cpm.ForceSplit(*split))
    assert (sim.tree_depth()["max_depth"] > 4 + 4) == dense  # 8^4 cells hold a particle each
    c = sim.counters()
    assert (c["leaf_pairs"], c["node_accepts"]) == (pairs, accepts)
    sim.close()
