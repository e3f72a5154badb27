"""The launch choices that a simulation reports are those it runs, and none of them changes a result beyond what the
header says."""
import numpy as np
import pytest

from test_gpu_walk import BOX, dense

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,team", [(20000, 4), (113665, 2), (227329, 1)])
@pytest.mark.parametrize("kind", ["uniform", "dense"])
def test_walk_groups(cpm, n, team, kind):
    """Sizes at which 4, 2 and 1 warps walk a group; dense boxes leave the groups to the ordered walk, and one
    particle outside the box takes their groups back."""
    x = dense(n) if kind == "dense" else np.random.default_rng(2).uniform(0, BOX, (n, 3)).astype(np.float32) % np.float32(BOX)
    sim = cpm.Simulation(cpm.Cosmology(0.0, 0.3, 0.7, 70.0), BOX, 32, x, np.zeros_like(x), 0.5,
                         cpm.ForceSplit(0.2, 0.8, 0.02, 0.5))
    t = sim.tuning()
    assert t["walk_warps"] in [w for w in (2, 4, 8) if w >= team]
    assert all(t["ms"][f"walk_warps{w}"] > 0.0 for w in (2, 4, 8))
    for out in (False, True):
        y = x.copy()
        if out:
            y[n // 2] -= np.float32(BOX)
        accs, pairs = [], []
        for warps in (4, 2, 8):
            sim.set_tuning(8, 1024, warps)
            assert sim.tuning()["walk_warps"] == max(warps, team)
            sim.set_state(y, np.zeros_like(y))
            accs.append(sim.state()["acc"])
            c = sim.counters()
            pairs.append((c["leaf_pairs"], c["node_accepts"], c["candidates"]))
        assert np.abs(accs[0]).max() > 0 and pairs[0] == pairs[1] == pairs[2]
        assert np.array_equal(accs[0], accs[1]) and np.array_equal(accs[0], accs[2])
    sim.close()


def test_times_of_fft_plans(cpm):
    """Plan 0 is plan 8: it has no time of its own, and takes the same steps."""
    import ctypes as C

    x = np.random.default_rng(4).uniform(0, BOX, (4096, 3)).astype(np.float32) % np.float32(BOX)
    sim = cpm.Simulation(cpm.Cosmology(0.0, 0.3, 0.7, 70.0), BOX, 48, x, np.zeros_like(x), 0.5, None)
    ms = np.full(9, -1.0, np.float32)
    cpm._native.check(cpm._native.lib().cpm_sim_autotune_report(sim.h, None, None, None, C.c_void_p(ms.ctypes.data)), sim=True)
    assert ms[0] > 0 and ms[1] > 0 and ms[2] == 0
    assert "fft_warp" not in sim.tuning()["ms"] and len(sim.tuning()["ms"]) == 8
    sim.close()


@pytest.mark.parametrize("mesh", [256, 512])
def test_fft_plans_of_large_meshes(cpm, mesh):
    """Plan 4 against plan 8, whose Poisson solve is checked against the oracle at these sizes: the PM forces agree to
    FFT rounding, about 1e-6 at these sizes; plan 0 gives those of plan 8 bit for bit."""
    x = np.random.default_rng(5).uniform(0, BOX, (mesh ** 3 // 64, 3)).astype(np.float32) % np.float32(BOX)
    sim = cpm.Simulation(cpm.Cosmology(0.0, 0.3, 0.7, 70.0), BOX, mesh, x, np.zeros_like(x), 0.5, None,
                         flags=cpm._native.SIM_NO_AUTOTUNE)
    acc = {}
    for plan in (8, 4, 0):
        sim.set_tuning(plan, 1024, 4)
        sim.set_state(x, np.zeros_like(x))
        acc[plan] = sim.state()["acc"].astype(np.float64)
    assert 0 < np.sqrt(((acc[4] - acc[8]) ** 2).sum() / (acc[8] ** 2).sum()) < 4e-6
    assert np.array_equal(acc[0], acc[8])
    sim.close()
