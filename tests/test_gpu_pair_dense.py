"""Dense scenes with each chunk split over a CTA pair, against the oracle bit for bit.

The pair's two tiles overlap by the rows that the rules of both halves reach, and a half
looks ten rows down for the friction of its sand: into rows that the other half updates.
Liquid that dries up in the first rows below the chunk's middle turns those rows to AIR in
the first sub-phase after that look.
"""
import numpy as np
import pytest

from helpers import compare_particles, compare_states, material_types
from oracle.binding import ORDER_PART
from test_gpu_dense_scenes import _scene

pytestmark = pytest.mark.gpu


def _steps(fse, oracle_mod, world, planes, chunk, seed, f32, shape, steps):
    types = material_types(fse)
    world.set_launch(shape)
    world.upload(planes)
    ow = oracle_mod.OracleWorld(world.width, world.height, chunk, 3, seed)
    ow.set_f32(f32)
    ow.set_state(world.state())
    for t in range(steps):
        world.step(1)
        ow.step(1, ORDER_PART)
        what = "shape %d %dx%d step %d" % (shape, world.width, world.height, t)
        compare_states(world.state(), ow.state(), types, what)
        compare_particles(world.particles(), ow.particles(), what)
    np.testing.assert_array_equal(world.ledger(), ow.ledger())
    world.close()


@pytest.mark.parametrize("shape", [2, 3])
@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("w,h,chunk,fire", [(132, 131, 128, False), (127, 260, 128, True), (70, 66, 64, True)])
def test_dense_scene_on_a_pair(fse, oracle_mod, w, h, chunk, fire, f32, shape):
    seed = w * 7 + h + chunk
    world = fse.World(w, h, chunk_size=chunk, seed=seed, f32_fluid=f32)
    _steps(fse, oracle_mod, world, _scene(fse, w, h, seed, f32, fire), chunk, seed, f32, shape, 3)


@pytest.mark.parametrize("shape", [2, 3])
@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("w,h,chunk", [(512, 512, 128), (130, 64, 64)])
def test_drying_below_the_middle(fse, oracle_mod, w, h, chunk, f32, shape):
    """Stopped sand above the middle, liquid that dries up within the step below it."""
    seed = 900 + w + chunk
    rng = np.random.default_rng(seed)
    sand, water, air = (fse.material_find(n) for n in ("GENERIC_SAND", "WATER", "GENERIC_AIR"))
    rows = np.arange(h) % chunk - chunk // 2  # 0: the first row below the middle
    top, wet = (rows >= -10) & (rows < 0), (rows >= 0) & (rows < 10)
    ids = np.full((h, w), fse.material_find("STONE"), np.uint16)
    r = rng.random((h, w))
    ids[top] = np.where(r < 0.6, sand, air)[top]
    ids[wet] = np.where(r < 0.8, water, sand)[wet]
    # 0.0004 and 0.0001 dry up; the others stay
    amount = rng.choice([0.0004, 0.0001, 0.9], (h, w), p=[0.5, 0.3, 0.2])
    sc = amount.astype(np.float32).view(np.int32) if f32 else (amount * 65536).astype(np.int32)
    planes = {"id": ids, "colour": np.where(ids == air, 0, rng.integers(0, 1 << 32, (h, w))).astype(np.uint32),
              "scalar": np.where(ids == water, sc, 0).astype(np.int32), "flags": np.zeros((h, w), np.uint8),
              "diff": np.zeros((h, w), np.int32)}
    world = fse.World(w, h, chunk_size=chunk, seed=seed, f32_fluid=f32)
    _steps(fse, oracle_mod, world, planes, chunk, seed, f32, shape, 2)
