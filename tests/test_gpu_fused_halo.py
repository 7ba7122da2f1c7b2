"""The fused tick's exchange of chunk borders inside one launch.

A chunk-pass stages its tile by tensor copies, which read what other CTAs of the same
launch wrote with ordinary stores a moment before. Small chunks make most of every tile a
border, and many worlds of one launch start each chunk-pass as soon as its neighbours are
done: the planes must equal those of one launch per pass, in which no such read happens.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,chunk,f32", [(512, 256, 16, False), (260, 516, 32, True), (1024, 512, 128, False)])
def test_borders_within_one_launch(fse, w, h, chunk, f32):
    worlds = []
    for shape in (0, 4):
        world = fse.World(w, h, chunk_size=chunk, seed=w + chunk, f32_fluid=f32)
        world.generate(fse.GEN_MIX, 3)
        world.set_launch(shape)
        worlds.append(world)
    for t in range(12):
        for world in worlds:
            world.step(2)
        a, b = (world.state() for world in worlds)
        for k in a:
            np.testing.assert_array_equal(a[k], b[k], "plane %s after %d steps" % (k, 2 * t + 2))
        assert worlds[0].particles().tobytes() == worlds[1].particles().tobytes()
    for world in worlds:
        world.close()


def test_borders_of_many_worlds_in_one_launch(fse):
    both = []
    for shape in (0, 4):
        worlds = []
        for k in range(48):
            world = fse.World(128 + 4 * (k % 7), 96 + 5 * (k % 5), chunk_size=32, seed=k)
            world.generate(fse.GEN_MIX, k)
            worlds.append(world)
        batch = fse.Batch(worlds)
        batch.set_launch(shape, 0)
        batch.step(10)
        both.append([world.state() for world in worlds])
        batch.close()
        for world in worlds:
            world.close()
    for a, b in zip(*both):
        for k in a:
            np.testing.assert_array_equal(a[k], b[k])
