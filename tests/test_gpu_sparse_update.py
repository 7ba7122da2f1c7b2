"""Few particles in large worlds, and block maps of every width, against the oracle.

The particle update takes its blocks from the population and from the size of the worlds'
block maps, and reads a block's row of materials at once where the width allows it.
"""
import numpy as np
import pytest

from helpers import compare_particles, compare_states, material_types
from oracle.binding import ORDER_PART

pytestmark = pytest.mark.gpu


def _falling(fse, n, w, h, seed):
    rng = np.random.default_rng(seed)
    p = np.zeros(n, fse.PARTICLE_DTYPE)
    p["x"], p["y"] = rng.uniform(0, w, n), rng.uniform(h * 0.4, h * 0.5 - 1, n)
    p["vx"], p["vy"], p["ay"] = rng.normal(0, 1, n), rng.uniform(1, 9, n), 0.1
    p["id"] = rng.choice([fse.material_find(m) for m in ("GENERIC_SAND", "WATER")], n)
    p["scalar"] = np.where(p["id"] == fse.material_find("WATER"), 65536, 0)
    p["fade_time"] = 60
    return p


# one block; blocks by the map (4,096 marks each: 64 rows of 64 blocks of cells and more);
# blocks by the population; widths that are and are not multiples of eight
@pytest.mark.parametrize("w,h,n", [(8, 64, 40), (9, 64, 40), (504, 520, 300), (1024, 512, 900), (1023, 520, 900),
                                   (1024, 1024, 1100), (2050, 1030, 60)])
def test_falling_particles_match_oracle(fse, oracle_mod, w, h, n):
    types = material_types(fse)
    ids = np.full((h, w), fse.material_find("STONE"), np.uint16)
    ids[h // 4:h // 2] = fse.material_find("GENERIC_AIR")
    ids[h // 2:h // 2 + 3, ::3] = fse.material_find("GENERIC_AIR")  # pits that fill up
    z = np.zeros((h, w), np.int32)
    world = fse.World(w, h, seed=n, particle_capacity=1 << 16)
    world.upload({"id": ids, "colour": z.view(np.uint32), "scalar": z, "flags": np.zeros((h, w), np.uint8), "diff": z})
    ow = oracle_mod.OracleWorld(w, h, 128, 3, n)
    ow.set_state(world.state())
    p = _falling(fse, n, w, h, n)
    world.addCell(p)
    ow.set_particles(p)
    for t in range(4):
        world.step(1)
        ow.step(1, ORDER_PART)
        compare_states(world.state(), ow.state(), types, "%dx%d step %d" % (w, h, t))
        compare_particles(world.particles(), ow.particles(), "%dx%d step %d" % (w, h, t))
    assert world.particle_count() < n
    world.close()


def test_batch_of_large_and_small_worlds(fse):
    """The marks of all worlds with particles count; worlds without any do not."""
    sizes = [(2048, 1024, 50), (64, 64, 0), (1000, 1000, 0), (520, 72, 400), (1600, 1600, 3)]
    both = []
    for batched in (False, True):
        worlds = []
        for k, (w, h, n) in enumerate(sizes):
            world = fse.World(w, h, seed=k, particle_capacity=1 << 17)
            world.generate(fse.GEN_MIX, k)
            if n:
                world.addCell(_falling(fse, n, w, h, k))
            worlds.append(world)
        if batched:
            batch = fse.Batch(worlds)
            batch.step(3)
            batch.close()
        else:
            for world in worlds:
                world.step(3)
        both.append([(world.state(), world.particles().tobytes()) for world in worlds])
        for world in worlds:
            world.close()
    for (a, pa), (b, pb) in zip(*both):
        assert pa == pb
        for k in a:
            np.testing.assert_array_equal(a[k], b[k])
