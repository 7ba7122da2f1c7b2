"""A batch as large as fse_batch_create accepts ticks like its worlds do one by one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MOST = 4095  # the worlds of one launch


def _particles(fse, n, seed):
    rng = np.random.default_rng(seed)
    p = np.zeros(n, fse.PARTICLE_DTYPE)
    p["x"], p["y"] = rng.uniform(0, 16, n), rng.uniform(0, 16, n)
    p["vx"], p["vy"], p["ay"] = rng.normal(0, 1, n), rng.normal(0, 1, n), 0.1
    p["id"], p["colour"] = fse.material_find("GENERIC_SAND"), 0xFFFFFFFF
    return p


def _world(fse, k):
    return fse.World(16, 16, chunk_size=16, seed=k, particle_capacity=512)


def test_the_largest_batches_tick(fse):
    """From the first size whose tables need more than the default shared memory up."""
    worlds = [_world(fse, k) for k in range(MOST)]
    looked_at = (0, 1, 777, 3890, 3891, MOST - 1)
    twins = {k: _world(fse, k) for k in looked_at}
    for k, twin in twins.items():
        for world in (worlds[k], twin):
            world.generate(fse.GEN_MIX, k)
            world.addCell(_particles(fse, 40, k))
    landed = 0
    for n in (3891, 3892, 4063, MOST):
        batch = fse.Batch(worlds[:n])
        batch.step(2)
        batch.close()
        for k, twin in twins.items():
            if k >= n:
                continue
            twin.step(2)
            a, b = worlds[k].state(), twin.state()
            for plane in a:
                np.testing.assert_array_equal(a[plane], b[plane], "%d worlds, world %d, %s" % (n, k, plane))
            assert worlds[k].particles().tobytes() == twin.particles().tobytes()
            landed += twin.particle_count() < 40
    assert landed > 0
    for world in worlds + list(twins.values()):
        world.close()
