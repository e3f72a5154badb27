"""Host outputs whose pages the library backs before it copies: never-touched, unaligned and pinned
buffers of sizes around its pieces (256 KB, 1 MB) get the same bytes, and nothing beside them changes."""
import ctypes as C
import mmap

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_side", [27, 28, 43, 45, 57])  # 12 n bytes: below and above 256 KB, 1 MB and 2 MB
def test_state_into_any_buffer(cpm, n_side):
    import torch
    rng = np.random.default_rng(n_side)
    n, box = n_side ** 3, float(n_side)
    x = rng.uniform(0, box, (n, 3)).astype(np.float32) % np.float32(box)
    sim = cpm.Simulation(cpm.Cosmology(0.0, 0.3, 0.7, 70.0), box, 32, x, np.zeros_like(x), 0.5, None)
    sim.step_to(0.52)
    want = sim.state()
    size = 12 * n

    def get(xa, pa, aa):
        cpm._native.check(cpm._native.lib().cpm_sim_get_state(sim.h, C.c_void_p(xa), C.c_void_p(pa), C.c_void_p(aa),
                                                              None, None), sim=True)

    for shift in (0, 4, 4092):
        raw = mmap.mmap(-1, 3 * size + 8 * 4096)  # pages never touched
        whole = np.frombuffer(raw, np.uint8)
        at = [4096 + shift + k * size for k in range(3)]
        whole[at[0] - 1] = whole[at[2] + size] = 0xA5
        base = whole.ctypes.data
        get(*(base + o for o in at))
        for o, key in zip(at, ("x", "p", "acc")):
            assert whole[o:o + size].tobytes() == want[key].tobytes()
        assert whole[at[0] - 1] == whole[at[2] + size] == 0xA5
        assert not whole[:at[0] - 1].any() and not whole[at[2] + size + 1:].any()
    pinned = torch.empty((3, n, 3), dtype=torch.float32).pin_memory()
    get(*(pinned[k].data_ptr() for k in range(3)))
    for k, key in enumerate(("x", "p", "acc")):
        assert np.array_equal(pinned[k].numpy(), want[key])
    sim.close()


def test_no_thread_starts_for_a_buffer_whose_pages_are_there(cpm):
    """Reading into arrays that were written before: the time of a read was up to a quarter longer for threads with
    nothing to do. Thread ids are given in turn, so the next one tells how many started (other processes' come
    on top); a read into untouched pages does start some."""
    import threading

    def next_id():
        ids = []
        t = threading.Thread(target=lambda: ids.append(threading.get_native_id()))
        t.start()
        t.join()
        return ids[0]

    n = 45 ** 3
    x = np.random.default_rng(1).uniform(0, 45, (n, 3)).astype(np.float32) % np.float32(45)
    sim = cpm.Simulation(cpm.Cosmology(0.0, 0.3, 0.7, 70.0), 45.0, 32, x, np.zeros_like(x), 0.5, None)

    def reads(buffers):
        before = next_id()
        for b in buffers:
            for _ in range(60 // len(buffers)):
                cpm._native.check(cpm._native.lib().cpm_sim_get_state(sim.h, C.c_void_p(b), None, None, None, None), sim=True)
        return next_id() - before

    used = np.ones((n, 3), np.float32)
    maps = [mmap.mmap(-1, 12 * n) for _ in range(60)]
    fresh = [np.frombuffer(m, np.uint8).ctypes.data for m in maps]
    assert reads([used.ctypes.data]) < 40 < 60 <= reads(fresh)
    assert np.array_equal(used, np.frombuffer(maps[-1], np.float32).reshape(n, 3))
    sim.close()
