"""The device memory that the particle read-out and the body calls use is given back.

What a world keeps is what a server's budget counts; a call's own workspace comes from
memory that all worlds share and that stays small however many of them make such calls.
"""
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SHARED = 64 << 20  # what stays between calls
SLACK = 16 << 20   # claims of the body calls and allocation granularity


def _records(fse, n, seed):
    rng = np.random.default_rng(seed)
    p = np.zeros(n, fse.PARTICLE_DTYPE)
    p["x"], p["y"] = rng.uniform(0, 64, n), rng.uniform(0, 64, n)
    p["lifetime"] = rng.integers(0, 1 << 30, n)
    p["id"] = fse.material_find("GENERIC_SAND")
    return p


def _bodies(fse, n, side, seed):
    rng = np.random.default_rng(seed)
    b = np.zeros(n, fse.BODY_DTYPE)
    b["w"] = b["h"] = side
    b["x"], b["y"] = rng.uniform(0, 190, n), rng.uniform(0, 190, n)
    b["cos_a"] = 1.0
    b["id"] = fse.material_find("GENERIC_OBJECT")
    return b


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_reads_and_bodies_of_many_worlds_keep_little(fse):
    """24 worlds with 200,000 particles (12 MB of records) and 100 boxes (8 MB of tiles)."""
    n, worlds = 200000, []
    p = _records(fse, n, 1)
    for k in range(24):
        worlds.append(fse.World(256, 256, seed=k, particle_capacity=n))
        worlds[-1].addCell(p)
    before = _free()
    for world in worlds:
        assert world.particles().tobytes() == p.tobytes()
    assert before - _free() <= SHARED + SLACK
    for world in worlds:
        b = _bodies(fse, 100, 64, 2)
        world.object_stamp(b)
        world.object_readback(b)
    assert before - _free() <= SHARED + SLACK
    worlds[0].trim()
    assert before - _free() <= SLACK
    for world in worlds:
        world.close()


def test_reads_of_served_worlds_stay_in_the_budget(fse):
    srv = fse.Server(4 << 30, 64)
    slots = [srv.add_world(256, 256, fse.GEN_MIX, k, seed=k, particle_capacity=200000) for k in range(24)]
    p = _records(fse, 150000, 3)
    for slot in slots:
        srv.world(slot).addCell(p)
    counted, before = srv.bytes_in_use(), _free()
    for slot in slots:
        assert srv.world(slot).particles().tobytes() == p.tobytes()
    assert before - _free() <= srv.bytes_in_use() - counted + SHARED + SLACK
    srv.close()


@pytest.mark.parametrize("cap", [1, 2047, 5000])
def test_reads_of_a_growing_population(fse, cap):
    """Around the number of records that every world holds, full and cut off by `cap`."""
    world = fse.World(64, 64, particle_capacity=1 << 16)
    want = np.zeros(0, fse.PARTICLE_DTYPE)
    for k, n in enumerate((1, 2046, 1, 1, 2046, 1, 3000)):
        p = _records(fse, n, k)
        world.addCell(p)
        want = np.concatenate([want, p])
        assert world.particles().tobytes() == want.tobytes()
        out, got = np.zeros(cap, fse.PARTICLE_DTYPE), fse.C.c_int(0)
        assert fse.lib().fse_particles_read(world.h, out.ctypes.data, cap, fse.C.byref(got)) == 0
        m = min(cap, len(want))
        assert got.value == len(want) and out[:m].tobytes() == want[:m].tobytes() and not out[m:].view(np.uint8).any()
    world.close()


def test_threads_share_the_memory(fse):
    """Reads and body calls of eight worlds at once, each world in a thread of its own."""
    n, wrong = 50000, []
    worlds = [fse.World(256, 256, seed=k, particle_capacity=1 << 18) for k in range(8)]
    single = fse.World(256, 256, seed=0, particle_capacity=1 << 18)
    single.addCell(_records(fse, n, 0))
    def boxes():  # side by side: all of their tiles find their own cells
        b = _bodies(fse, 36, 32, 5)
        b["x"], b["y"] = (np.arange(36) % 6) * 32, (np.arange(36) // 6) * 32
        return b

    b = boxes()
    single.object_stamp(b)
    assert single.object_readback(b) == 36 * 32 * 32
    state = single.state()

    def work(world):
        try:
            p = _records(fse, n, 0)
            world.addCell(p)
            for _ in range(20):
                if world.particles().tobytes() != p.tobytes():
                    wrong.append("records")
                c = boxes()
                world.object_stamp(c)
                world.object_readback(c)
                if c.tobytes() != b.tobytes():
                    wrong.append("bodies")
        except Exception as e:  # noqa: BLE001
            wrong.append(repr(e))

    threads = [threading.Thread(target=work, args=(world,)) for world in worlds]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    for world in worlds:
        got = world.state()
        for k in state:
            np.testing.assert_array_equal(got[k], state[k])
    for world in worlds + [single]:
        world.close()


def test_threads_read_one_world(fse):
    """Reads of different lengths of one world at the same time."""
    p, wrong = _records(fse, 6000, 4), []
    world = fse.World(64, 64, particle_capacity=1 << 16)
    world.addCell(p)

    def work(cap):
        for _ in range(100):
            out, got = np.zeros(cap, fse.PARTICLE_DTYPE), fse.C.c_int(0)
            st = fse.lib().fse_particles_read(world.h, out.ctypes.data, cap, fse.C.byref(got))
            if st != 0 or out.tobytes() != p[:cap].tobytes():
                wrong.append(cap)

    threads = [threading.Thread(target=work, args=(cap,)) for cap in (1, 100, 2000, 2048, 2049, 6000)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    world.close()
